// How many producer warps may share a ring of shared-memory stages (tc_gemm.cu).
//
// The k-blocks go round the producers, and a producer waits only in its own turns, by parity: before k-block kb it asks
// for the release of kb - stages, and a parity answers that question only once kb - 2 * stages has been released (before
// that the barrier's previous phase has the same parity, and the wait returns at once over a stage in use).  What a
// producer knows is its own last turn: kb - producers - stages was released.  So producers <= stages.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define VAICU_HOST_DEVICE __host__ __device__
#else
#define VAICU_HOST_DEVICE
#endif

namespace vaicu {

// One thread takes 600-800 cycles to wait for a stage, announce its bytes and issue its two or three copies (170 + 35 + 200
// each, measured), longer than the MMAs of most tiles and than HBM needs for a stage: three of them keep up.
constexpr uint32_t kTcProducers = 3;

VAICU_HOST_DEVICE constexpr uint32_t tc_producers(uint32_t stages) { return stages < kTcProducers ? stages : kTcProducers; }

}  // namespace vaicu
