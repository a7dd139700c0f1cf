// Row-wise top-k sampling over logits [M, N]: vAi's TopKSampling node
// (vai/nodes/topk-sampling.h:9-31, vai/shaders/topk-sampling.comp):
//   out[i] = sample(softmax(top-k(I[i, :]) / temperature), u)
// with the reference's exact rules: candidates ranked by (value descending, index
// ascending); Z and the running sum accumulated in that order in fp32 with the row maximum
// subtracted; the first rank whose running sum reaches u * Z is the sample (rank 0 if none).
//
// Two launches, as in the reference.  Popping the best k times costs k dependent rounds of shuffles, so both
// stages select by rank instead: a lower bound T on the k-th best is cheap (the k-th best of a few hundred maxima), few
// entries reach it, and each of those counts how many outrank it - its place.
// Stage 1: block (g, row) owns a 2048-column slice, 8 columns per thread; T is the k-th best of the 256 threads' maxima,
// at most 8 k columns reach it.  Stage 2: T is the k-th best of the first ceil(k / G) entries of the G sorted lists.
// Where more than 1024 entries reach that T (the winners crowd in a few slices) one warp merges the sorted lists.
// Rows of at most 2048 columns need stage 1's block only.  Both steps are exact: the top-k of a union is within
// the union of the parts' top-k.  u lives in device memory so that a recorded launch sees each step's value.
#include "common.cuh"

namespace vaicu {

namespace {

constexpr uint32_t kList = 8;             // columns per thread
constexpr uint32_t kMaxK = 128;           // vAi TopKSampling::maxK
constexpr uint32_t kPartThreads = 256;    // stage 1: 256 * 8 = 2048 columns per block
constexpr uint32_t kSlice = kPartThreads * kList;
constexpr uint32_t kMaxKept = kMaxK * kList;   // entries that can reach stage 1's bound; stage 2's limit
constexpr float kLowest = -3.4028235e38f; // the shader's sentinel (finite: softmax terms stay NaN-free)

__device__ __forceinline__ bool outranks(float av, uint32_t ai, float bv, uint32_t bi)
{
    return av > bv || (av == bv && ai < bi);
}

// The same order as one integer: larger is better.  NaN and what is below the sentinel rank with it (never chosen).
typedef unsigned long long Key;
constexpr Key kNone = 0;
__device__ __forceinline__ Key rank_key(float v, uint32_t i)
{
    if (!outranks(v, i, kLowest, 0xFFFFFFFFu)) return kNone;
    const uint32_t b = __float_as_uint(v + 0.0f);                  // -0 and +0 are equal: the index decides
    return ((Key)(b & 0x80000000u ? ~b : b | 0x80000000u) << 32) | (Key)(~i);
}
// Entries of list[0, n) that outrank key.
__device__ __forceinline__ uint32_t count_above(const Key* list, uint32_t n, Key key)
{
    uint32_t c = 0;
#pragma unroll 8
    for (uint32_t i = 0; i < n; ++i) c += list[i] > key ? 1u : 0u;
    return c;
}

struct TopkParams {
    const void* logits;       // stage 1: [M, N] of dtype
    const uint2* cand_in;     // stage 2: [M, G * k] (value bits, index), G sorted lists of k
    uint2* cand_out;          // stage 1 with G > 1: [M, G * k]
    uint32_t* out;            // sampling launch: [M]
    const float* u;           // device scalar in [0, 1)
    uint32_t N;               // stage 1: row width; stage 2: lists per row (G)
    uint32_t k;               // min(K, row width of the logits)
    int32_t dtype;
    float temperature;
    // vocabulary slabs: the logits are a window of wider rows / the candidates carry global indices
    size_t ld;                // stage 1: elements between rows of the logits
    uint32_t index_base;      // stage 1: added to every column index
    // stage 2 reads list l of row r at cand_in[l * list_stride + r * row_stride] (entries)
    size_t list_stride, row_stride;
    uint32_t list_len;        // entries per list in cand_in (>= k; the tail may be padding)
    uint2* list_out;          // stage 2: write the merged, sorted k_out entries per row here instead of sampling
    uint32_t k_out;           // entries per row in list_out (>= k: the tail is padded with sentinels)
};

// One warp merges `nlists` descending lists of `len` (value, index) entries each, stored
// back to back at `lists`, into the best `k` of their union, in order, at top_v / top_i.
// Lane l walks lists l, l + 32, ...: their heads live in registers, SLOTS lists per lane at most.
template <uint32_t SLOTS>
__device__ __forceinline__ void merge_lists(const uint2* lists, uint32_t nlists, size_t stride, uint32_t len, uint32_t k, float* top_v,
                                            uint32_t* top_i, uint32_t lane)
{
    float hv[SLOTS];
    uint32_t hi[SLOTS], pos[SLOTS];
#pragma unroll
    for (uint32_t j = 0; j < SLOTS; ++j) {
        const uint32_t l = lane + 32u * j;
        pos[j] = 0u;
        if (l < nlists && len > 0u) {
            const uint2 c = lists[(size_t)l * stride];
            hv[j] = __uint_as_float(c.x); hi[j] = c.y;
        } else {
            hv[j] = kLowest; hi[j] = 0xFFFFFFFFu;
        }
    }
    for (uint32_t r = 0; r < k; ++r) {
        // this lane's best head, then the warp's
        float bv = hv[0];
        uint32_t bi = hi[0];
#pragma unroll
        for (uint32_t j = 1; j < SLOTS; ++j)
            if (outranks(hv[j], hi[j], bv, bi)) { bv = hv[j]; bi = hi[j]; }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, off);
            const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
            if (outranks(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (lane == 0u) { top_v[r] = bv; top_i[r] = bi; }
        // the list whose head won advances (indices are unique, sentinels aside)
#pragma unroll
        for (uint32_t j = 0; j < SLOTS; ++j) {
            if (hi[j] == bi && hv[j] == bv && bi != 0xFFFFFFFFu) {
                const uint32_t l = lane + 32u * j;
                if (++pos[j] < len) {
                    const uint2 c = lists[(size_t)l * stride + pos[j]];
                    hv[j] = __uint_as_float(c.x); hi[j] = c.y;
                } else {
                    hv[j] = kLowest; hi[j] = 0xFFFFFFFFu;
                }
            }
        }
    }
    __syncwarp();
}

// Temperature softmax over the k winners and the inverse-CDF sample (topk-sampling.comp:237-258).  Called by all
// threads of a block; the exponentials are taken side by side (into `terms`), the sums run in rank order.
__device__ __forceinline__ void sample(const float* top_v, const uint32_t* top_i, float* terms, uint32_t k, float temperature, float u,
                                       uint32_t* out)
{
    const float inv_t = 1.0f / fmaxf(temperature, 1e-6f);
    const float m = top_v[0];
    for (uint32_t r = threadIdx.x; r < k; r += blockDim.x) terms[r] = expf((top_v[r] - m) * inv_t);
    __syncthreads();
    if (threadIdx.x != 0u) return;
    float z = 0.0f;
    for (uint32_t r = 0; r < k; ++r) z += terms[r];
    const float target = u * z;
    float cum = 0.0f;
    uint32_t pick = top_i[0];
    for (uint32_t r = 0; r < k; ++r) {
        cum += terms[r];
        if (cum >= target) { pick = top_i[r]; break; }
    }
    *out = pick;
}

// What the block keeps while it selects.
struct Kept {
    Key key[kMaxKept];
    float val[kMaxKept];
    Key best[kPartThreads];
    float top_v[kMaxK];
    uint32_t top_i[kMaxK];
    float terms[kMaxK];
    Key bound;
    uint32_t count;
};

// The kept entries in rank order, the tail filled with sentinels.  All threads.
__device__ __forceinline__ void place_by_rank(Kept& s, uint32_t count, uint32_t k)
{
    for (uint32_t c = threadIdx.x; c < count; c += kPartThreads) {
        const Key key = s.key[c];
        const uint32_t r = count_above(s.key, count, key);
        if (r < k) { s.top_v[r] = s.val[c]; s.top_i[r] = ~(uint32_t)key; }
    }
    for (uint32_t r = count + threadIdx.x; r < k; r += kPartThreads) { s.top_v[r] = kLowest; s.top_i[r] = 0xFFFFFFFFu; }
    __syncthreads();
}

// Stage 1.  SAMPLE: the row fits one block, which also samples.
template <bool SAMPLE>
__global__ void __launch_bounds__(kPartThreads) topk_slice_kernel(const TopkParams p)
{
    const uint32_t row = blockIdx.y, g = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    __shared__ Kept s;
    dependency_wait();
    launch_dependents();         // behind the wait: a Linear after this may request weights that a launch ahead has written
    const uint32_t slice = (p.N + G - 1u) / G;
    const uint32_t s0 = g * slice, s1 = (s0 + slice < p.N) ? s0 + slice : p.N;
    float v[kList];
    Key key[kList], best = kNone;
#pragma unroll
    for (uint32_t j = 0; j < kList; ++j) {
        const uint32_t i = s0 + tid + j * kPartThreads;
        v[j] = i < s1 ? load_as_f32(p.logits, p.dtype, (size_t)row * p.ld + i) : kLowest;
    }
#pragma unroll
    for (uint32_t j = 0; j < kList; ++j) {
        const uint32_t i = s0 + tid + j * kPartThreads;
        key[j] = i < s1 ? rank_key(v[j], p.index_base + i) : kNone;
        best = key[j] > best ? key[j] : best;
    }
    s.best[tid] = best;
    if (tid == 0u) { s.bound = kNone; s.count = 0u; }
    __syncthreads();
    // keys of columns differ, so at most one thread is k-th; with fewer than k threads that hold any, all entries are kept
    if (best != kNone && count_above(s.best, kPartThreads, best) == p.k - 1u) s.bound = best;
    __syncthreads();
    const Key bound = s.bound;
#pragma unroll
    for (uint32_t j = 0; j < kList; ++j)
        if (key[j] != kNone && key[j] >= bound) {
            const uint32_t at = atomicAdd(&s.count, 1u);
            s.key[at] = key[j];
            s.val[at] = v[j];
        }
    __syncthreads();
    place_by_rank(s, s.count, p.k);
    if (SAMPLE) {
        sample(s.top_v, s.top_i, s.terms, p.k, p.temperature, *p.u, p.out + row);
    } else if (p.list_out) {
        // the row fits this block and its sorted list is the result: k entries, then padding
        for (uint32_t r = tid; r < p.k_out; r += kPartThreads)
            p.list_out[(size_t)row * p.k_out + r] = r < p.k ? make_uint2(__float_as_uint(s.top_v[r]), s.top_i[r])
                                                           : make_uint2(__float_as_uint(kLowest), 0xFFFFFFFFu);
    } else {
        for (uint32_t r = tid; r < p.k; r += kPartThreads)
            p.cand_out[((size_t)row * G + g) * p.k + r] = make_uint2(__float_as_uint(s.top_v[r]), s.top_i[r]);
    }
}

// Stage 2: one block per row over its G <= 256 sorted lists.
__global__ void __launch_bounds__(kPartThreads) topk_merge_kernel(const TopkParams p)
{
    const uint32_t row = blockIdx.x, tid = threadIdx.x, G = p.N;
    __shared__ Kept s;
    dependency_wait();
    launch_dependents();         // behind the wait: a Linear after this may request weights that a launch ahead has written
    const uint2* lists = p.cand_in + (size_t)row * p.row_stride;
    // the bound: the first entries of the lists, k of them where the lists are that long, at most 256: one per thread
    const uint32_t even = (p.k + G - 1u) / G, ahead = even < p.list_len ? even : p.list_len;
    Key mine = kNone;
    if (tid < G * ahead) {
        const uint2 c = lists[(size_t)(tid / ahead) * p.list_stride + tid % ahead];
        mine = rank_key(__uint_as_float(c.x), c.y);
    }
    s.best[tid] = mine;
    if (tid == 0u) { s.bound = kNone; s.count = 0u; }
    __syncthreads();
    if (mine != kNone && count_above(s.best, kPartThreads, mine) == p.k - 1u) s.bound = mine;
    __syncthreads();
    const Key bound = s.bound;
    for (uint32_t i = tid; i < G * p.list_len; i += kPartThreads) {
        const uint2 c = lists[(size_t)(i / p.list_len) * p.list_stride + i % p.list_len];
        const Key key = rank_key(__uint_as_float(c.x), c.y);
        if (key != kNone && key >= bound) {
            const uint32_t at = atomicAdd(&s.count, 1u);
            if (at < kMaxKept) { s.key[at] = key; s.val[at] = __uint_as_float(c.x); }
        }
    }
    __syncthreads();
    if (s.count <= kMaxKept) {
        place_by_rank(s, s.count, p.k);
    } else {
        if (tid < 32u) merge_lists<8>(lists, G, p.list_stride, p.list_len, p.k, s.top_v, s.top_i, tid);
        __syncthreads();
    }
    if (p.list_out) {
        for (uint32_t r = tid; r < p.k_out; r += kPartThreads)
            p.list_out[(size_t)row * p.k_out + r] = r < p.k ? make_uint2(__float_as_uint(s.top_v[r]), s.top_i[r])
                                                           : make_uint2(__float_as_uint(kLowest), 0xFFFFFFFFu);
    } else {
        sample(s.top_v, s.top_i, s.terms, p.k, p.temperature, *p.u, p.out + row);
    }
}

}  // namespace

// Blocks per row in stage 1 (1: single launch).
uint32_t topk_groups(uint32_t N) { return (N + kSlice - 1u) / kSlice; }

namespace {
// Stage 2 over the lists of each row; samples into `out`, or writes the merged list to `list_out`.
cudaError_t launch_merge(const TopkParams& q, uint32_t M, cudaStream_t stream)
{
    return launch_pdl(topk_merge_kernel, dim3(M), dim3(kPartThreads), 0, stream, q);
}
}  // namespace

// `list_out` null: the TopKSampling node (sample into `out`).  `list_out` set: the per-slab step of a
// vocabulary-split head — the sorted top-K list of each row of this slab, indices offset by index_base.
cudaError_t launch_topk(const void* logits, int dtype, uint32_t M, uint32_t N, size_t ld, uint32_t K, uint32_t index_base,
                        float temperature, const float* u, void* workspace, uint32_t* out, void* list_out, cudaStream_t stream)
{
    TopkParams p{};
    p.logits = logits; p.dtype = dtype; p.temperature = temperature; p.u = u; p.out = out;
    p.N = N;
    p.ld = ld;
    p.index_base = index_base;
    p.k = K < N ? K : N;
    p.list_out = reinterpret_cast<uint2*>(list_out);
    p.k_out = K;
    const uint32_t G = topk_groups(N);
    if (G == 1u) {
        return list_out ? launch_pdl(topk_slice_kernel<false>, dim3(1, M), dim3(kPartThreads), 0, stream, p)
                        : launch_pdl(topk_slice_kernel<true>, dim3(1, M), dim3(kPartThreads), 0, stream, p);
    }
    p.cand_out = reinterpret_cast<uint2*>(workspace);
    p.list_out = nullptr;                       // the slices feed stage 2
    cudaError_t e = launch_pdl(topk_slice_kernel<false>, dim3(G, M), dim3(kPartThreads), 0, stream, p);
    if (e != cudaSuccess) return e;
    TopkParams q = p;
    q.logits = nullptr;
    q.cand_in = reinterpret_cast<const uint2*>(workspace);
    q.cand_out = nullptr;
    q.N = G;
    q.list_len = p.k;
    q.list_stride = p.k;
    q.row_stride = (size_t)G * p.k;
    q.list_out = reinterpret_cast<uint2*>(list_out);
    return launch_merge(q, M, stream);
}

cudaError_t launch_topk_sample(const void* logits, int dtype, uint32_t M, uint32_t N, uint32_t K, float temperature,
                               const float* u, void* workspace, uint32_t* out, cudaStream_t stream)
{
    return launch_topk(logits, dtype, M, N, N, K, 0u, temperature, u, workspace, out, nullptr, stream);
}

// Merge step of a vocabulary-split head: `groups` sorted lists per row (one per GPU, list_len entries each,
// padding allowed at the tail), list g of row m at pairs[g * group_stride + m * list_len]; keeps the best k
// of their union and samples.
cudaError_t launch_topk_merge_sample(const void* pairs, uint32_t groups, size_t group_stride, uint32_t M, uint32_t list_len,
                                     uint32_t k, float temperature, const float* u, uint32_t* out, cudaStream_t stream)
{
    TopkParams q{};
    q.cand_in = reinterpret_cast<const uint2*>(pairs);
    q.N = groups;
    q.k = k;
    q.list_len = list_len;
    q.list_stride = group_stride;
    q.row_stride = list_len;
    q.temperature = temperature;
    q.u = u;
    q.out = out;
    return launch_merge(q, M, stream);
}

}  // namespace vaicu
