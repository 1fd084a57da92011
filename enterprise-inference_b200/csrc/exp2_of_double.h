// 2^x for x <= 0 as an fp32 number, from an exponent held in 64 bits (host and device: its error is tested on the CPU).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define B200_HD __host__ __device__ __forceinline__
#else
#define B200_HD inline
#endif

namespace b200 {

// Beside its last rounding to 2^-24.5 of itself (q's roundings): n = x rounded, 2^f = 1 + f q(f) on |f| <= 1/2 by its Taylor series (terms ln2^k / k!, the
// first left out 5e-9).  (The argument of an expf would be rounded first: half an ulp of the weight for each unit of it.)  Below -120 it is 0, -inf too; NaN goes on.
B200_HD float exp2_of_double(double x) {
  if (x < -120.0) return 0.f;
  const double u = x + 6755399441055744.0;        // 1.5 * 2^52: n in the low bits
  const float f = (float)(x - (u - 6755399441055744.0));
  float q = 1.52527338e-5f;
  q = fmaf(q, f, 1.54035304e-4f);
  q = fmaf(q, f, 1.33335581e-3f);
  q = fmaf(q, f, 9.61812911e-3f);
  q = fmaf(q, f, 5.55041087e-2f);
  q = fmaf(q, f, 2.40226507e-1f);
  q = fmaf(q, f, 6.93147181e-1f);
#ifdef __CUDA_ARCH__
  const float p = __int_as_float((127 + __double2loint(u)) << 23);
#else
  int64_t bits;
  std::memcpy(&bits, &u, 8);
  const uint32_t e = (uint32_t)(127 + (int32_t)bits) << 23;
  float p;
  std::memcpy(&p, &e, 4);
#endif
  return fmaf(f, q, 1.0f) * p;
}

}  // namespace b200
