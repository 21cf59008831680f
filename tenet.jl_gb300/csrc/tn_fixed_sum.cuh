// Sums of FP64 values over a warp or CTA in fixed point: integer additions and the warp's redux
// take 4 to 30 clocks where a DADD takes 64.
#pragma once

#include <cuda_runtime.h>

// Every lane's value is cut towards zero to 55 bits below 2^(emax − 1022), emax the largest exponent
// field of the warp.  A unit is 2^(emax − 1077), the largest value at least 2^(emax − 1023): a cut is less
// than 2⁻⁵⁴ of it, and the 31 others' cuts of a warp less than 31·2⁻⁵⁴ (a value within a factor of 4
// of the largest is not cut at all).  An FP64 tree's five roundings are 2⁻⁵³ of the partial sums each: less
// where one value outweighs the rest, more where the values are alike.  Values below FP64's normal
// range count as zero.  The parts of 24 bits add up without a carry between them; four warps' sums
// aligned to a common exponent fit in 63 bits.
__device__ __forceinline__ unsigned exponent_field(double v) { return ((unsigned)__double2hiint(v) >> 20) & 0x7ff; }
__device__ __forceinline__ long long fixed_warp_sum(double v, unsigned emax) {
  const int hi = __double2hiint(v);
  const unsigned e = exponent_field(v);
  unsigned long long b = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 34) | ((unsigned long long)(unsigned)__double2loint(v) << 2);
  b = e ? b >> min(emax - e, 63u) : 0ull;
  const long long sg = hi >> 31, f = ((long long)b ^ sg) - sg;
  const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)f & 0xffffffu);
  const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(f >> 24) & 0xffffffu);
  const int top = __reduce_add_sync(0xffffffffu, (int)(f >> 48));
  return ((long long)top << 48) + ((long long)mid << 24) + (long long)lo;
}
// the sum of four warps' sums (16-byte aligned) and their exponents; E: the common one
__device__ __forceinline__ long long fixed_sum4(const long long* part, const int* exps, int& E) {
  const int4 ew = *reinterpret_cast<const int4*>(exps);
  E = max(max(ew.x, ew.y), max(ew.z, ew.w));
  return ((part[0] >> min(E - ew.x, 63)) + (part[1] >> min(E - ew.y, 63))) +
         ((part[2] >> min(E - ew.z, 63)) + (part[3] >> min(E - ew.w, 63)));
}
// T·2^(E − 1077); a sum with an infinity or a NaN in it (E = 0x7ff) is NaN
__device__ __forceinline__ double fixed_value(long long T, int E) {
  const double v = (double)T;
  const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff, r = ex + E - 1077;
  if (E == 0x7ff) return __longlong_as_double(0x7ff8000000000000ll);
  if (ex == 0) return 0.0;
  if (r < 1 || r > 2046) return ldexp(v, E - 1077);
  return __hiloint2double(hi + ((E - 1077) << 20), __double2loint(v));
}
// |T| < 2⁶³ as a float
__device__ __forceinline__ float fixed_to_float(long long T) {
  const unsigned long long A = T < 0 ? (unsigned long long)-T : (unsigned long long)T;
  const float f = fmaf((float)(unsigned)(A >> 32), 4294967296.f, (float)(unsigned)A);
  return T < 0 ? -f : f;
}
