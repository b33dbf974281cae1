// How the warps of a row tile share their two buffers in nvfp4_a16_kernel: plain C++, compiled for the GPU by
// nvfp4_a16.cu and for the host by tests/test_a16_exchange_cpu.py.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define MUSER_A16_HD __host__ __device__ __forceinline__
#else
#define MUSER_A16_HD inline
#endif

namespace muser {

// In a step every warp writes its contributions to one buffer, all meet at a barrier, and all read that buffer.  A warp
// that is ahead writes the next step's buffer while others still read this one's, and writes this one's again only
// behind the next barrier, for which every warp must have finished reading: safe as long as no two steps in a row use
// the same buffer.  So the steps are counted through all passes of a call (a pass takes 2 * PAIRS tokens): counted from
// zero in each, a pass of an odd number of steps would end on the buffer that the next one starts with.
MUSER_A16_HD uint32_t a16_buffer(uint32_t pass, uint32_t steps_per_pass, uint32_t step) { return (pass * steps_per_pass + step) & 1u; }

} // namespace muser
