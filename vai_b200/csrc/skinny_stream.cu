// Linear with 5 to 8 rows of activations and 16-bit weights, up to some 70 MB of them (skinny_stream_fits): the streaming decode form (gemv_stream.cuh) with its dot
// products on mma.sync.
//
// At these sizes the layer is still bound by the bytes of its weights (8 rows: 8 MACs per weight), but one
// FMA per weight and row is more than the FMA units deliver at HBM speed, and the tcgen05 kernel pays for its
// launches instead: a cast of the activations, a K split over CTAs, a fold.  m16n8k16 fits the batch exactly
// (16 weight rows x 8 activation rows), needs no tensor memory and no descriptors, and lets one launch do all of
// it: the block converts the activations into fragments once and keeps them in registers (8 warps split K, 4096 of
// K at a time), weights come through the lanes' FIFOs, which do not wait for the launch ahead, and the warps' partial
// sums are added up in shared memory.  Llama-3.2-1B step at 8 rows, 16 blocks: 930 -> 710 us (11 -> 4 launches a block).
//
// A lane's FIFO vectors are its own MMA fragments: four k-pairs of two MMAs are 8 consecutive elements of its row, and
// the activations are taken in the same order (the order of k inside a dot product is free).
#include <type_traits>

#include "gemv_stream.cuh"

namespace vaicu {

namespace {

constexpr uint32_t kTileRows = 16;                       // weight rows per MMA tile (8 gate + 8 value rows with a gate)
constexpr uint32_t kChunk = 512;                         // elements of K per step: 64 per warp
constexpr uint32_t kBatchTiles = 2;                      // tiles between two folds
constexpr uint32_t kSumPitch = 20;                       // floats between two activation rows of a tile's sums
constexpr uint32_t kTileSums = 8u * kSumPitch;
constexpr uint32_t kSkinnySmem = kStreamFifoBytes + 8u * kBatchTiles * kTileSums * 4u;
constexpr uint32_t kStep = 4;                            // vectors per lane and chunk: two k-halves of rows g and g + 8
constexpr uint32_t kSteps = kStreamDepth / kStep;

template <typename TW> __device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma16816<__half>(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma16816<__nv_bfloat16>(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Eight consecutive activations as 16-bit pairs of the weights' type (fp32 ones rounded, as the tcgen05 path's cast does;
// without XA those may begin at any element).
template <typename TW, bool XA> __device__ __forceinline__ uint4 load_x8(const LinearArgs& a, size_t at)
{
    if (a.i_dtype != VAICU_DTYPE_F32) return *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.I) + at);
    const float* s = reinterpret_cast<const float*>(a.I) + at;
    float4 lo, hi;
    if constexpr (XA) {
        lo = reinterpret_cast<const float4*>(s)[0];
        hi = reinterpret_cast<const float4*>(s)[1];
    } else {
        lo = make_float4(s[0], s[1], s[2], s[3]);
        hi = make_float4(s[4], s[5], s[6], s[7]);
    }
    uint4 o;
    if constexpr (std::is_same<TW, __half>::value) {
        __half2 h0 = __floats2half2_rn(lo.x, lo.y), h1 = __floats2half2_rn(lo.z, lo.w);
        __half2 h2 = __floats2half2_rn(hi.x, hi.y), h3 = __floats2half2_rn(hi.z, hi.w);
        o.x = *reinterpret_cast<uint32_t*>(&h0); o.y = *reinterpret_cast<uint32_t*>(&h1);
        o.z = *reinterpret_cast<uint32_t*>(&h2); o.w = *reinterpret_cast<uint32_t*>(&h3);
    } else {
        __nv_bfloat162 h0 = __floats2bfloat162_rn(lo.x, lo.y), h1 = __floats2bfloat162_rn(lo.z, lo.w);
        __nv_bfloat162 h2 = __floats2bfloat162_rn(hi.x, hi.y), h3 = __floats2bfloat162_rn(hi.z, hi.w);
        o.x = *reinterpret_cast<uint32_t*>(&h0); o.y = *reinterpret_cast<uint32_t*>(&h1);
        o.z = *reinterpret_cast<uint32_t*>(&h2); o.w = *reinterpret_cast<uint32_t*>(&h3);
    }
    return o;
}

// SC: chunks of K whose activations are held in registers at a time.  Order of work: batches of tiles; per batch, spans
// of SC chunks; per span the batch's tiles; per tile the span's chunks.
// XA: the activations are 16-byte aligned.
template <typename TW, int SC, bool XA>
__global__ void __launch_bounds__(kStreamThreads, 2) skinny_stream_kernel(const StreamParams p)
{
    extern __shared__ __align__(128) uint8_t smem[];
    float* sums = reinterpret_cast<float*>(smem + kStreamFifoBytes);       // [tile][warp][activation row][weight row]

    const LinearArgs& a = p.a;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const bool gate = a.gate_fuse != 0;
    const uint32_t K = a.K, H = p.H, M = a.M, row_bytes = K * 2u;
    const uint32_t T = gate ? kTileRows / 2u : kTileRows;        // output columns per tile
    const uint32_t u0 = (uint32_t)((uint64_t)H * blockIdx.x / gridDim.x), u1 = (uint32_t)((uint64_t)H * (blockIdx.x + 1u) / gridDim.x);
    const uint32_t chunks = (K + kChunk - 1u) / kChunk;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t k_lane = warp * 64u + t * 8u;                 // this lane's first element of a chunk; the second half is 32 on

    // The loader's place: tile at lj of the batch at lb, chunk lc of the span at ls.
    const uint32_t fifo = (uint32_t)__cvta_generic_to_shared(smem) + threadIdx.x * 16u;
    uint32_t lb = u0, lj = u0, ls = 0, lc = 0, lslot = 0;
    const uint8_t *src_lo = nullptr, *src_hi = nullptr;          // this lane's two rows of the tile; null past the range
    bool trigger = true;
    auto set_rows = [&]() {
        const uint32_t lo = lj + g, hi = gate ? H + lj + g : lj + 8u + g;
        src_lo = lo < u1 ? stream_row(p, lo, row_bytes) : nullptr;
        src_hi = (gate ? lo < u1 : hi < u1) ? stream_row(p, hi, row_bytes) : nullptr;
    };
    set_rows();
    auto load_step = [&]() {
        if (lb < u1) {
#pragma unroll
            for (uint32_t h = 0; h < 2u; ++h) {
                const uint32_t k = lc * kChunk + k_lane + h * 32u;
                const bool in = k < K;
                const uint32_t at = fifo + (lslot * kStep + 2u * h) * (kStreamThreads * 16u);
                const bool lo = in && src_lo != nullptr, hi = in && src_hi != nullptr;
                fifo_load(at, lo ? (const void*)(src_lo + k * 2u) : a.W, lo ? 16u : 0u);
                fifo_load(at + kStreamThreads * 16u, hi ? (const void*)(src_hi + k * 2u) : a.W, hi ? 16u : 0u);
            }
            if (++lc == chunks || lc == ls + SC) {
                lj += T;
                const uint32_t end = lb + kBatchTiles * T < u1 ? lb + kBatchTiles * T : u1;
                if (lj >= end) {
                    if (lc == chunks) { lb = end; ls = 0; } else { ls = lc; }
                    lj = lb;
                }
                lc = ls;
                set_rows();
            }
        } else if (trigger) {
            trigger = false;
            launch_dependents();       // the last load is on its way: the next launch's blocks may move in
        }
        fifo_commit();                 // (an empty group past the end keeps the count)
        if (++lslot == kSteps) lslot = 0;
    };
#pragma unroll 1
    for (uint32_t i = 0; i + 1u < kSteps; ++i) load_step();

    const EpilogueArgs ep = make_epilogue_args(a);
    uint32_t slot = 0;
    uint4 xb[SC][2];
    dependency_wait();
    for (uint32_t b0 = u0; b0 < u1; b0 += kBatchTiles * T) {
        const uint32_t b1 = b0 + kBatchTiles * T < u1 ? b0 + kBatchTiles * T : u1;
        for (uint32_t c0 = 0; c0 < chunks; c0 += SC) {
            if (chunks > SC || b0 == u0) {
#pragma unroll
                for (int c = 0; c < SC; ++c)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t k = (c0 + c) * kChunk + k_lane + h * 32u;
                        xb[c][h] = (g < M && k < K) ? load_x8<TW, XA>(a, (size_t)g * K + k) : make_uint4(0, 0, 0, 0);
                    }
            }
            uint32_t tile = 0;
            for (uint32_t j = b0; j < b1; j += T, ++tile) {
                float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
                for (int c = 0; c < SC; ++c) {
                    if (c0 + c >= chunks) break;
                    load_step();
                    fifo_wait<(int)kSteps - 1>();
                    uint4 w[kStep];
#pragma unroll
                    for (uint32_t i = 0; i < kStep; ++i) w[i] = fifo_read(fifo + (slot * kStep + i) * (kStreamThreads * 16u));
                    if (++slot == kSteps) slot = 0;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint4 lo = w[2 * h], hi = w[2 * h + 1];
                        mma16816<TW>(acc[0], lo.x, hi.x, lo.y, hi.y, xb[c][h].x, xb[c][h].y);
                        mma16816<TW>(acc[1], lo.z, hi.z, lo.w, hi.w, xb[c][h].z, xb[c][h].w);
                    }
                }
                float* d = sums + (size_t)(tile * 8u + warp) * kTileSums + 2u * t * kSumPitch + g;
                const float v[4] = {acc[0][0] + acc[1][0], acc[0][1] + acc[1][1], acc[0][2] + acc[1][2], acc[0][3] + acc[1][3]};
                float* const at[4] = {d, d + kSumPitch, d + 8, d + kSumPitch + 8};
#pragma unroll
                for (int e = 0; e < 4; ++e) *at[e] = c0 == 0u ? v[e] : *at[e] + v[e];
            }
        }
        __syncthreads();
        // add up the warps and finish the batch's outputs; neighbouring threads take neighbouring columns
        const uint32_t width = b1 - b0;
        for (uint32_t e = threadIdx.x; e < width * M; e += kStreamThreads) {
            const uint32_t m = e / width, u = e - m * width, tile = u / T, r = u - tile * T;
            const float* s = sums + (size_t)tile * 8u * kTileSums + m * kSumPitch + r;
            const uint32_t n = b0 + u;
            const size_t flat = (size_t)m * H + n;
            const float bias = gate || p.nseg ? 0.0f : read_bias(ep, flat), res = gate || p.nseg ? 0.0f : read_res(ep, flat);
            float v = 0.0f, up = 0.0f;
#pragma unroll
            for (uint32_t w = 0; w < 8u; ++w) {
                v += s[w * kTileSums];
                if (gate) up += s[w * kTileSums + T];
            }
            if (gate) store_from_f32(a.O, a.o_dtype, flat, finish_gated(ep, v, up, n, H, flat));
            else if (p.nseg) store_segment(p, m, n, v);
            else store_from_f32(a.O, a.o_dtype, flat, finish_output_pre(ep, v, bias, res));
        }
        if (b1 < u1) __syncthreads();            // the sums are reused by the next batch
    }
}

template <typename TW, int SC, bool XA> cudaError_t launch_skinny_form(const StreamParams& p, int grid, cudaStream_t stream)
{
    auto kern = skinny_stream_kernel<TW, SC, XA>;
    static SmemOptIn optin;
    if (cudaError_t e = optin.ensure(kern, (int)kSkinnySmem, cudaSharedmemCarveoutMaxShared); e != cudaSuccess) return e;
    return launch_pdl(kern, dim3((unsigned)grid), dim3(kStreamThreads), kSkinnySmem, stream, p);
}
template <typename TW> cudaError_t launch_skinny_typed(const StreamParams& p, int grid, cudaStream_t stream)
{
    if ((reinterpret_cast<uintptr_t>(p.a.I) & 15u) == 0u)
        return p.a.K <= 4u * kChunk ? launch_skinny_form<TW, 4, true>(p, grid, stream) : launch_skinny_form<TW, 8, true>(p, grid, stream);
    return p.a.K <= 4u * kChunk ? launch_skinny_form<TW, 4, false>(p, grid, stream) : launch_skinny_form<TW, 8, false>(p, grid, stream);
}

}  // namespace

// Measured against the tcgen05 kernel (its cast, GEMM and fold) in recorded chains of 396 layers at 5 and 8 rows, bf16 and fp32
// activations, K 64 to 16384, 16 to 131072 weight rows; us at 8 rows, bf16, here / there:
//   * every pair of tiles ends in a fold during which the block multiplies nothing, so up to six tiles per block:
//     2048 x 8192 10.1 / 11.5, 4096 x 8192 (four) as fast, 2048 x 16384 (seven) 16.0 / 13.6, 2048 x 128256 103 / 79; seven while
//     a tile is short: 1024 x 16384 7.8 / 9.0, but 64 x 16384 (all fold) 5.5 / 3.9; and gated up to K = 2048: 2048 x 16384
//     15.7 / 15.1, but a recorded Llama-3.2-1B step with fp32 activations 708 / 749 (three launches more per block);
//   * beyond K = 4096 the activations leave the registers between two pairs of tiles: only layers of one tile per block, at least half
//     full: 8192 x 2048 9.5 / 10.9, 8192 x 2560 (two) 16.1 / 12.1, 8192 x 300 7.2 / 6.3, 12288 x 300 13.2 / 7.3.
// The choice is 0.6 % off the better of the two on average, 15 % at most.
bool skinny_stream_fits(uint32_t N, uint32_t K, bool gate, int sm_count)
{
    const uint32_t H = gate ? N / 2u : N, tile = gate ? kTileRows / 2u : kTileRows;
    const uint32_t cols = (H + (uint32_t)sm_count - 1u) / (uint32_t)sm_count, tiles = (cols + tile - 1u) / tile;
    if (K <= 4096u) return tiles <= (K >= 256u && K <= (gate ? 2048u : 1536u) ? 7u : 6u);
    return K <= 8192u && tiles == 1u && cols * 2u >= tile;
}

cudaError_t launch_skinny_stream(const LinearArgs& a, int sm_count, uint32_t nseg, const uint32_t* rows, const void* const* w,
                                 void* const* o, cudaStream_t stream)
{
    if (a.M == 0u || a.M > kSkinnyStreamRows || a.K % 8u) return cudaErrorInvalidValue;
    StreamParams p{};
    p.a = a;
    p.H = a.gate_fuse ? a.N / 2u : a.N;
    if (cudaError_t e = stream_segments(p, nseg, rows, w, o); e != cudaSuccess) return e;
    const int grid = (int)(p.H < (uint32_t)sm_count ? p.H : (uint32_t)sm_count);
    if (a.w_dtype == VAICU_DTYPE_F16) return launch_skinny_typed<__half>(p, grid, stream);
    if (a.w_dtype == VAICU_DTYPE_BF16) return launch_skinny_typed<__nv_bfloat16>(p, grid, stream);
    return cudaErrorInvalidValue;
}

}  // namespace vaicu
