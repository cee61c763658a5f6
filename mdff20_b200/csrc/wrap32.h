// Differences of 32-bit fixed-point fractions of the box (units of 2^-32): modulo 2^32, which is
// the minimum image.  About half of the differences across the box edge leave the range of int, so
// they are formed unsigned.
#pragma once

#ifdef __CUDACC__
#define MDFF_WRAP_HD __host__ __device__ __forceinline__
#else
#define MDFF_WRAP_HD inline
#endif

namespace mdffgpu {

MDFF_WRAP_HD int wrap_diff(int a, int b) { return (int)((unsigned)a - (unsigned)b); }

}  // namespace mdffgpu
