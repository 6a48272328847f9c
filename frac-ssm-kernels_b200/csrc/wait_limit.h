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
}  // namespace fracssm
#undef FRACSSM_HD
