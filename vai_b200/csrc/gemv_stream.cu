// Kernel and planning of the streaming decode form; see gemv_stream.cuh.
#include "gemv_stream.cuh"

namespace vaicu {

namespace {

template <typename T> struct Vec { static constexpr int N = 8; };
template <> struct Vec<float> { static constexpr int N = 4; };

template <typename TW> __device__ __forceinline__ void unpack_w(const uint4& v, float2* f);
template <> __device__ __forceinline__ void unpack_w<float>(const uint4& v, float2* f)
{
    f[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
    f[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w));
}
template <> __device__ __forceinline__ void unpack_w<__half>(const uint4& v, float2* f)
{
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
}
template <> __device__ __forceinline__ void unpack_w<__nv_bfloat16>(const uint4& v, float2* f)
{
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
}

// N consecutive activations from element `at` (at % N == 0, 16-byte aligned matrix) as float2 pairs.
template <int N> __device__ __forceinline__ void load_x(const LinearArgs& a, size_t at, float2* xf)
{
    if (a.i_dtype == VAICU_DTYPE_F32) {
        const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.I) + at);
#pragma unroll
        for (int q = 0; q < N / 4; ++q) {
            const float4 t = s[q];
            xf[2 * q] = make_float2(t.x, t.y);
            xf[2 * q + 1] = make_float2(t.z, t.w);
        }
        return;
    }
    uint32_t w[N / 2];
    const uint2* s = reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(a.I) + at);
#pragma unroll
    for (int q = 0; q < N / 4; ++q) { const uint2 t = s[q]; w[2 * q] = t.x; w[2 * q + 1] = t.y; }
    if (a.i_dtype == VAICU_DTYPE_F16) {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) xf[i] = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    } else {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) xf[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u));
    }
}

constexpr uint32_t kPartFloats = 2048;           // partial sums held between two folds
constexpr uint32_t kGemvStreamSmem = kStreamFifoBytes + kPartFloats * 4u;

// XV: 16-byte weight vectors per lane and row.  A block's rows are taken in rounds of 8 / ks, one row per group of ks
// warps; with a gate a warp alternates between the gate and the value row of its output column.
template <typename TW, int XV, bool ARGMAX>
__global__ void __launch_bounds__(kStreamThreads, 2) gemv_stream_kernel(const StreamParams p)
{
    constexpr int VEC = Vec<TW>::N, PAIRS = VEC / 2;
    constexpr uint32_t STEP = XV <= 5 ? XV : XV / 2;             // vectors requested, awaited and multiplied together
    constexpr uint32_t STEPS = kStreamDepth / STEP;              // ... and as many such steps under way
    constexpr uint32_t PER_ROW = XV / STEP;
    static_assert(XV % STEP == 0, "whole steps");
    extern __shared__ __align__(128) uint8_t smem[];
    float* part = reinterpret_cast<float*>(smem + kStreamFifoBytes);       // [row][ks]

    const LinearArgs& a = p.a;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const bool gate = a.gate_fuse != 0;
    const uint32_t K = a.K, H = p.H;
    const uint32_t row_bytes = K * (uint32_t)sizeof(TW);
    const uint32_t u0 = (uint32_t)((uint64_t)H * blockIdx.x / gridDim.x), u1 = (uint32_t)((uint64_t)H * (blockIdx.x + 1u) / gridDim.x);
    const uint32_t KS = p.ks, RG = kStreamWarps / KS;
    const uint32_t rg = warp / KS, ks = warp % KS;
    const uint32_t nvec = K / VEC, v0 = ks * 32u + lane, vstep = KS * 32u;

    // The loader's place: unit `lu`, its value row next when lval, step `ls` of that row; `slot` wraps with the FIFO.
    const uint32_t fifo = (uint32_t)__cvta_generic_to_shared(smem) + threadIdx.x * 16u;
    uint32_t lu = u0 + rg, ls = 0, lslot = 0;
    bool lval = false, trigger = true;
    auto load_step = [&]() {
        if (lu < u1) {
            const uint8_t* src = stream_row(p, lval ? H + lu : lu, row_bytes);
#pragma unroll
            for (uint32_t i = 0; i < STEP; ++i) {
                const uint32_t v = v0 + (ls * STEP + i) * vstep;
                fifo_load(fifo + (lslot * STEP + i) * (kStreamThreads * 16u), src + (v < nvec ? v : 0u) * 16u, v < nvec ? 16u : 0u);
            }
            if (++ls == PER_ROW) {
                ls = 0;
                if (gate && !lval) lval = true;
                else { lval = false; lu += RG; }
            }
        } else if (trigger) {
            trigger = false;
            launch_dependents();       // this warp's last load is on its way: the next launch's blocks may move in
        }
        fifo_commit();                 // (an empty group past the end keeps the count)
        if (++lslot == STEPS) lslot = 0;
    };
#pragma unroll 1
    for (uint32_t i = 0; i + 1u < STEPS; ++i) load_step();

    const EpilogueArgs ep = make_epilogue_args(a);
    float am_best = kArgmaxLowest;
    uint32_t am_at = 0xFFFFFFFFu;

    dependency_wait();
    float2 xf[XV][PAIRS];
#pragma unroll
    for (int i = 0; i < XV; ++i) {
        const uint32_t v = v0 + (uint32_t)i * vstep;
        if (v < nvec) load_x<VEC>(a, (size_t)v * VEC, xf[i]);
        else
#pragma unroll
            for (int e = 0; e < PAIRS; ++e) xf[i][e] = make_float2(0.0f, 0.0f);
    }
    // bias and residual of this thread's first output, requested ahead of the products
    float early_bias = 0.0f, early_res = 0.0f;
    const bool early = !gate && !p.nseg && threadIdx.x < (u1 - u0 < p.batch ? u1 - u0 : p.batch);
    if (early) {
        const size_t flat = u0 + threadIdx.x;
        early_bias = read_bias(ep, flat);
        early_res = read_res(ep, flat);
    }

    uint32_t slot = 0;
    for (uint32_t b0 = u0; b0 < u1; b0 += p.batch) {
        const uint32_t b1 = b0 + p.batch < u1 ? b0 + p.batch : u1;
        for (uint32_t u = b0 + rg; u < b1; u += RG) {
            for (uint32_t half = 0; half < (gate ? 2u : 1u); ++half) {
                float2 acc[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
                for (uint32_t s = 0; s < PER_ROW; ++s) {
                    load_step();
                    fifo_wait<(int)STEPS - 1>();
                    uint4 wv[STEP];
#pragma unroll
                    for (uint32_t i = 0; i < STEP; ++i) wv[i] = fifo_read(fifo + (slot * STEP + i) * (kStreamThreads * 16u));
                    if (++slot == STEPS) slot = 0;
#pragma unroll
                    for (uint32_t i = 0; i < STEP; ++i) {
                        float2 wf[PAIRS];
                        unpack_w<TW>(wv[i], wf);
#pragma unroll
                        for (int e = 0; e < PAIRS; ++e) acc[e & 1] = __ffma2_rn(wf[e], xf[s * STEP + i][e], acc[e & 1]);
                    }
                }
                float v = (acc[0].x + acc[0].y) + (acc[1].x + acc[1].y);
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
                if (lane == 0u) part[((u - b0) + half * p.batch) * KS + ks] = v;
            }
        }
        __syncthreads();
        // fold the warps of each row and finish the batch's outputs
        for (uint32_t u = threadIdx.x; u < b1 - b0; u += kStreamThreads) {
            const uint32_t n = b0 + u;
            float v = 0.0f, up = 0.0f;
            for (uint32_t s = 0; s < KS; ++s) {
                v += part[u * KS + s];
                if (gate) up += part[(p.batch + u) * KS + s];
            }
            if (gate) {
                store_from_f32(a.O, a.o_dtype, n, finish_gated(ep, v, up, n, H, n));
            } else if (p.nseg) {
                store_segment(p, 0u, n, v);
            } else {
                const float o = (early && n == u0 + threadIdx.x) ? finish_output_pre(ep, v, early_bias, early_res) : finish_output(ep, v, n);
                if (!ARGMAX || p.am.write_logits) store_from_f32(a.O, a.o_dtype, n, o);
                // the Argmax node reads the stored logits: compare what the store would hold
                if (ARGMAX) argmax_take(round_through(a.o_dtype, o), p.am.index_base + n, am_best, am_at);
            }
        }
        if (b1 < u1) __syncthreads();            // part is reused by the next batch
    }

    if constexpr (ARGMAX) {
        // the block's candidate, then the last block to take a ticket folds all of them; nobody waits
        __shared__ float s_val[kStreamWarps];
        __shared__ uint32_t s_at[kStreamWarps];
        __shared__ bool s_last;
        auto warp_best = [&](float& best, uint32_t& at) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, off);
                const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, at, off);
                argmax_take(ov, oi, best, at);
            }
        };
        warp_best(am_best, am_at);
        if (lane == 0u) { s_val[warp] = am_best; s_at[warp] = am_at; }
        __syncthreads();
        if (threadIdx.x == 0u) {
            for (uint32_t w = 1; w < kStreamWarps; ++w) argmax_take(s_val[w], s_at[w], am_best, am_at);
            p.am.block_val[blockIdx.x] = am_best;
            p.am.block_idx[blockIdx.x] = am_at;
            __threadfence();                           // the candidate is visible before the ticket
            s_last = atomicAdd(p.am.count, 1u) == gridDim.x - 1u;
        }
        __syncthreads();
        if (s_last && warp == 0u) {
            __threadfence();
            float best = kArgmaxLowest;
            uint32_t at = 0xFFFFFFFFu;
            for (uint32_t b = lane; b < gridDim.x; b += 32u) argmax_take(__ldcg(p.am.block_val + b), __ldcg(p.am.block_idx + b), best, at);
            warp_best(best, at);
            if (lane == 0u) {
                p.am.out_idx[0] = at == 0xFFFFFFFFu ? p.am.index_base : at;   // a row of NaNs: its first column
                if (p.am.out_val) p.am.out_val[0] = best;
                *p.am.count = 0u;                      // ready for the next launch
            }
        }
    }
}

template <typename TW, int XV, bool ARGMAX>
cudaError_t launch_stream_form(const StreamParams& p, int grid, cudaStream_t stream)
{
    auto kern = gemv_stream_kernel<TW, XV, ARGMAX>;
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(kern, (int)kGemvStreamSmem, cudaSharedmemCarveoutMaxShared); e != cudaSuccess) return e;
    return launch_pdl(kern, dim3((unsigned)grid), dim3(kStreamThreads), kGemvStreamSmem, stream, p);
}

template <typename TW, int XV>
cudaError_t launch_stream_one(const StreamParams& p, int grid, cudaStream_t stream)
{
    return p.am.out_idx ? launch_stream_form<TW, XV, true>(p, grid, stream) : launch_stream_form<TW, XV, false>(p, grid, stream);
}

template <typename TW>
cudaError_t launch_stream_typed(const StreamParams& p, int xv, int grid, cudaStream_t stream)
{
    switch (xv) {
    case 3: return launch_stream_one<TW, 3>(p, grid, stream);
    case 4: return launch_stream_one<TW, 4>(p, grid, stream);
    case 5: return launch_stream_one<TW, 5>(p, grid, stream);
    case 6: return launch_stream_one<TW, 6>(p, grid, stream);
    case 8: return launch_stream_one<TW, 8>(p, grid, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// Geometry of the streaming form; false where it does not apply: more than one row (with 2 to 4 the folds of every row's
// sums take longer than the loads: 2560 x 20480 bf16, 31 / 51 / 61 us against the register form's 21 / 25 / 30), K too long
// for the registers that hold the activations, and where the register form is the better one (here / there, us, in recorded
// chains of one layer, 700 layers, K 64 to 16384):
//   * above 140 MB, where the hand-over no longer counts and the register form keeps 128 KB per SM on their way instead of 96:
//     201 MB layers 33.6 / 33.6 (1536 x 65536), 44.1 / 36.8 (5000 x 20000), 148 MB 36.0 / 27.3 (8200 x 9000); still ahead at
//     134 MB 21.3 / 24.1 (8192 x 8192) and 105 MB 17.5 / 19.8 (2560 x 20480);
//   * where K fills less than three quarters of the vectors that the lanes load, and a block has more than two rounds of
//     rows: 200 x 32768 10.5 / 6.8, 400 x 8192 4.1 / 3.2, 552 x 9000 4.3 / 3.9, but 200 x 768 (one round) 1.9 / 2.0.
// Of the layers that stay, most gain 5 to 30 %; the losses are up to 16 % at 8 to 13 MB, about one FIFO per SM (2048 x 2560 4.0 / 3.5,
// while 2560 x 2048 takes 3.5 / 4.0).
// The warps per row: the fewest rounds of rows per block, weighed by the vectors of a round and 1.5 for its fold.
bool choose_gemv_stream(const LinearArgs& a, int sm_count, GemvStream* out)
{
    GemvStream c{};
    const uint32_t esz = dtype_size(a.w_dtype), vec = 16u / esz;
    const uint32_t H = a.gate_fuse ? a.N / 2u : a.N;
    if (a.M != 1u || a.K % vec || H == 0u || (uint64_t)a.N * a.K * esz > 140000000ull) return false;
    const uint32_t nvec = a.K / vec, units = (H + (uint32_t)sm_count - 1u) / (uint32_t)sm_count;
    uint32_t ks = 0u;
    double best = 1e30;
    for (uint32_t k = 1u; k <= kStreamWarps; k *= 2u) {
        const uint32_t need = (nvec + 32u * k - 1u) / (32u * k);
        if (need > 8u) continue;
        const int xv = need <= 3u ? 3 : (need <= 6u ? (int)need : 8);        // the widths that are built
        const uint32_t rg = kStreamWarps / k, rounds = (units + rg - 1u) / rg;
        const double cost = rounds * (xv + 1.5);
        if (cost < best) { best = cost; ks = k; c.xv = xv; }
    }
    if (!ks) return false;
    c.ks = ks;
    const uint32_t rg = kStreamWarps / ks, slots = 32u * ks * (uint32_t)c.xv;
    if (nvec * 4u < slots * 3u && units > 2u * rg) return false;
    // whole rounds of the warps' row groups between two folds
    c.batch = kPartFloats / ((a.gate_fuse ? 2u : 1u) * ks) / rg * rg;
    c.grid = (int)(H < (uint32_t)sm_count ? H : (uint32_t)sm_count);
    *out = c;
    return true;
}

cudaError_t launch_gemv_stream(const LinearArgs& a, const GemvConfig& cfg, uint32_t nseg, const uint32_t* rows, const void* const* w,
                               void* const* o, const GemvArgmax* argmax, cudaStream_t stream)
{
    const GemvStream& c = cfg.stream;
    StreamParams p{};
    p.a = a;
    p.H = a.gate_fuse ? a.N / 2u : a.N;
    p.ks = c.ks; p.batch = c.batch;
    if (argmax) p.am = *argmax;
    if (cudaError_t e = stream_segments(p, nseg, rows, w, o); e != cudaSuccess) return e;
    switch (a.w_dtype) {
    case VAICU_DTYPE_F32: return launch_stream_typed<float>(p, c.xv, c.grid, stream);
    case VAICU_DTYPE_F16: return launch_stream_typed<__half>(p, c.xv, c.grid, stream);
    case VAICU_DTYPE_BF16: return launch_stream_typed<__nv_bfloat16>(p, c.xv, c.grid, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace vaicu
