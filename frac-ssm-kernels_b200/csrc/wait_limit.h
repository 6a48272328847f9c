// When a bounded device-side wait gives up.  Plain C++, so that it can be tested on the host.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define FRACSSM_HD __host__ __device__ __forceinline__
#else
#define FRACSSM_HD inline
#endif

namespace fracssm {
namespace umma {

// Whether a wait that began at `start` has used up its limit (below 2^63).  The difference is a signed number: a
// reading of the timer a tick before the start means that nothing has passed; as an unsigned number it would be 2^64 ns
// and the wait would give up at once.
FRACSSM_HD bool past_limit(uint64_t start, uint64_t now, uint64_t limit_ns) {
  return static_cast<int64_t>(now - start) > static_cast<int64_t>(limit_ns);
}

}  // namespace umma

// Blocks that share work with those that have started (csrc/decode_layers.cu).

// How long the first block keeps the list open while n of `blocks` have started: until the wait has cost as much as going without
// the others will, for work that takes all of them work_ns, and 10 us at least, which their start takes.
FRACSSM_HD uint64_t list_patience_ns(uint32_t n, uint32_t blocks, uint64_t work_ns) {
  return 10000 + work_ns * (blocks - n) / n;
}
// Limit of the waits among them: on top of `limit_ns` what one of them alone would take for the whole of it, since few may have
// started and the shares of two may be all and nothing.
FRACSSM_HD uint64_t list_limit_ns(uint32_t blocks, uint64_t work_ns, uint64_t limit_ns) { return limit_ns + work_ns * blocks; }

}  // namespace fracssm
#undef FRACSSM_HD
