// pm_fp.cuh — comparisons of FP64 values on their bits.  The FP64 pipe takes
// half a lane per cycle in each quarter of an SM, also for comparisons: a
// test for zero costs as much there as an FMA, and nothing on the integer
// pipe.
#ifndef PM_FP_CUH
#define PM_FP_CUH

#include <cuda_runtime.h>

namespace pm {

__device__ __forceinline__ bool nonzero(float v) { return v != 0.f; }
__device__ __forceinline__ bool nonzero(double v) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffll) != 0;
}

// |v| as a key that orders like it; a NaN compares below everything, as it
// does in "fabs(v) > best"
__device__ __forceinline__ float abs_key(float v) { return v == v ? fabsf(v) : -1.f; }
__device__ __forceinline__ long long abs_key(double v) {
  const long long b = __double_as_longlong(v) & 0x7fffffffffffffffll;
  return b <= 0x7ff0000000000000ll ? b : -1ll;
}
template <typename T>
struct KeyOf {
  typedef float type;
};
template <>
struct KeyOf<double> {
  typedef long long type;
};

}  // namespace pm

#endif
