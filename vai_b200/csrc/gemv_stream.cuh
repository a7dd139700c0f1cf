// Decode path of Linear, one row, in the form that keeps HBM busy across a chain of layers.
//
// One persistent block per SM takes a contiguous range of output columns.  Every lane keeps a FIFO of the 16-byte
// weight vectors that it alone will multiply, in shared memory: it requests them with cp.async, in the order of their
// use, and reads back only its own, so the loads need no barrier, no registers and no producer.  The activations stay
// in registers for the whole launch (lane l of the s-th warp of a row multiplies the same vectors of every row), the
// products are packed fp32 FMAs, each warp leaves one partial sum per row, and the block adds those up and stores
// its outputs, coalesced.
//
// What it is for: in a recorded step the register form (gemv.cu) lost 2.3 us per launch, because a block's loads
// started only when a block of the launch ahead had left its registers.  Here a block holds at most half of an
// SM's shared memory and asks for its successor (griddepcontrol.launch_dependents) when a warp has issued its LAST
// load: the next layer's first 96 KB per SM arrive while this layer is multiplied, folded and stored.
// Recorded one-row steps, register form -> this one: Llama-3.2-1B shapes 578 -> 519 us, Llama-3.2-3B blocks 1304 -> 1049,
// GPT-2-small 195 -> 167.
// Bulk copies into a ring with mbarriers were measured first: one thread issues a copy per 110 cycles and turns a stage
// round in 560, so stages below 16 KB cannot reach HBM speed (4.1 TB/s at 8 KB, 2.1 at 4 KB, of 6.65 at 16 KB).
#pragma once

#include "common.cuh"

namespace vaicu {

constexpr uint32_t kStreamThreads = 256;                         // 8 warps
constexpr uint32_t kStreamWarps = kStreamThreads / 32u;
constexpr uint32_t kStreamDepth = 24;                            // vectors per lane: 96 KB per block, two blocks per SM
constexpr uint32_t kStreamFifoBytes = kStreamDepth * kStreamThreads * 16u;

struct StreamParams {
    LinearArgs a;
    uint32_t H;              // output columns
    uint32_t ks;             // warps that share a row's K: 1, 2, 4 or 8
    uint32_t batch;          // units (output columns) between two folds
    uint32_t nseg;           // > 0: a group of plain Linears, as in gemv.cu
    uint32_t seg_begin[4];
    const void* seg_w[3];
    void* seg_o[3];
    GemvArgmax am;
};

// 16 bytes of weights into this lane's slot; bytes = 0 reads nothing and leaves zeros.
__device__ __forceinline__ void fifo_load(uint32_t slot, const void* src, uint32_t bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(slot), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fifo_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the newest N groups of this thread's copies have landed.
template <int N> __device__ __forceinline__ void fifo_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 fifo_read(uint32_t slot)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(slot) : "memory");
    return v;
}

// Weight row `row` of the layer, or of the group's members side by side.
__device__ __forceinline__ const uint8_t* stream_row(const StreamParams& p, uint32_t row, uint32_t row_bytes)
{
    const void* base = p.a.W;
    if (p.nseg) {
        const uint32_t sg = (row >= p.seg_begin[1] ? 1u : 0u) + (row >= p.seg_begin[2] ? 1u : 0u);
        base = p.seg_w[sg];
        row -= p.seg_begin[sg];
    }
    return reinterpret_cast<const uint8_t*>(base) + (size_t)row * row_bytes;
}

// Where output column n of activation row m of a group goes.
__device__ __forceinline__ void store_segment(const StreamParams& p, uint32_t m, uint32_t n, float v)
{
    const uint32_t sg = (n >= p.seg_begin[1] ? 1u : 0u) + (n >= p.seg_begin[2] ? 1u : 0u);
    const uint32_t width = p.seg_begin[sg + 1u] - p.seg_begin[sg];
    store_from_f32(p.seg_o[sg], p.a.o_dtype, (size_t)m * width + (n - p.seg_begin[sg]), v);
}

// The members of a group, side by side; nothing for a single Linear.
inline cudaError_t stream_segments(StreamParams& p, uint32_t nseg, const uint32_t* rows, const void* const* w, void* const* o)
{
    p.nseg = nseg;
    if (!nseg) return cudaSuccess;
    if (nseg < 2u || nseg > 3u) return cudaErrorInvalidValue;
    uint32_t total = 0;
    for (uint32_t i = 0; i < 4u; ++i) p.seg_begin[i] = 0xFFFFFFFFu;
    for (uint32_t i = 0; i < nseg; ++i) {
        p.seg_begin[i] = total;
        p.seg_w[i] = w[i];
        p.seg_o[i] = o[i];
        total += rows[i];
    }
    p.seg_begin[nseg] = total;
    return total == p.a.N ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace vaicu
