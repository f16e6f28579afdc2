// A particle row (x, y, z, m) of 32 bytes as one load: a gather then takes one
// sector look-up per lane instead of the two of a pair of 16-byte loads.  Rows
// are 32-byte aligned (device allocations) and not written by the kernel.
#pragma once
#include <cuda_runtime.h>

namespace ahop {

__device__ __forceinline__ double4 load_row(const double4* p) {
  double4 r;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
  return r;
}

}  // namespace ahop
