// FP64 building blocks of the Householder and LU kernels: reciprocal and
// reciprocal square root from short series, and the reflector made of them.
// Device code only, compiled by nvcc (cs_babd.cu) and by NVRTC (in front of
// cs_kernels.cuh).
#ifndef CS_FP64_CUH
#define CS_FP64_CUH

// -x as an integer operation (the compiler spends an FP64 add on it)
__device__ __forceinline__ double cs_neg(double x) {
  return __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x));
}

// 1 / p to the last bit or two: the reciprocal of the leading 23 bits in FP32,
// then one third-order step r (1 + e + e^2), e = 1 - p r, |e| < 2^-22 (the
// truncated geometric series for 1 / (1 - e)): 3 FP64 instructions where the
// division takes about 9, on the unit that bounds these kernels.  Exponents
// near the ends of the range (and 0, inf, NaN) divide.
__device__ __forceinline__ double cs_rcp(double p) {
  const int hi = __double2hiint(p), lo = __double2loint(p);
  const int ex = (hi >> 20) & 0x7ff;
  if (ex < 16 || ex > 2030) return 1.0 / p;
  // mantissa in [1, 2) as FP32, its reciprocal in (1/2, 1]
  const unsigned rf = __float_as_uint(__frcp_rn(__uint_as_float(0x3f800000u | ((unsigned)(hi & 0xfffff) << 3) | ((unsigned)lo >> 29))));
  // the FP32 number as FP64 bits, scaled by 2^(1023 - ex), with p's sign
  const int rex = (int)(rf >> 23) - 127 + 1023 + (1023 - ex);
  const double r = __hiloint2double((hi & 0x80000000) | (rex << 20) | (int)((rf >> 3) & 0xfffff), (int)(rf << 29));
  const double e = fma(-p, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// 1 / sqrt(x), x > 0, to the last bit or two: FP32 on the leading bits, then
// r (1 + h/2 + 3 h^2/8), h = 1 - x r^2, |h| < 2^-20 (the truncated binomial
// series of (1 - h)^(-1/2)): 5 FP64 instructions in a chain
__device__ __forceinline__ double cs_rsqrt(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int ex = (hi >> 20) & 0x7ff;
  if (hi < 0 || ex < 16 || ex > 2030) return 1.0 / sqrt(x);
  const int odd = (ex & 1) ^ 1;  // 1023 is odd: mantissa 2^odd in [1, 4)
  const float m = __uint_as_float(((unsigned)(127 + odd) << 23) | ((unsigned)(hi & 0xfffff) << 3) | ((unsigned)lo >> 29));
  const unsigned rf = __float_as_uint(rsqrtf(m));
  const int rex = (int)(rf >> 23) - 127 + 1023 - ((ex - 1023 - odd) >> 1);
  const double r = __hiloint2double((rex << 20) | (int)((rf >> 3) & 0xfffff), (int)(rf << 29));
  const double h = fma(-(x * r), r, 1.0);
  return fma(r, h * fma(0.375, h, 0.5), r);
}

// Householder reflector H = I - t v v^T of a column with sum of squares ss and
// leading entry x0: H column = g e_0 (the sign rule of
// matrix_factorization_cuda.py:37-54), v_0 = x0 - g, v the column below, and
// t = 2 / |v|^2 = 1 / (ss + |x0 g|).  False when |v|^2 / 2 is a number below
// `least` (the bits of a positive double; eps / 2 by default: nothing to
// eliminate).  A column with a NaN reflects, and so hands it on to every column:
// skipped, what it holds below the diagonal would be dropped and the solution
// would come out finite.
//
// a = ss r, r = ss^(-1/2), is sqrt(ss) to 2.5 of 2^-53; g takes a Newton step
// from it, a + (ss - a^2) r / 2, as exact as a rounded square root and beside the
// chain a, |v|^2 / 2, t (t to 3.3 of 2^-53).  A square root and two divisions
// before: with few merges in flight their latency (about 600 cycles each) was a
// third of a merge.  Its users form the products p_c = column . column c of the
// untouched columns first: p of the column itself is ss, and v . column c = p_c -
// g times the leading entry of column c, so one pass over the rows serves both.
__device__ __forceinline__ bool cs_reflector(double ss, double x0, double* g, double* v0, double* t,
                                             long long least = 0x3ca0000000000000ll) {
  const double r = cs_rsqrt(ss);
  const double a = ss * r;
  const double s = fma(fabs(x0), a, ss);  // |v|^2 / 2
  // (r / 2 by its exponent; where r is 0, infinite or a NaN so is a a NaN)
  const double w = fma(fma(-a, a, ss), __hiloint2double(__double2hiint(r) - (1 << 20), __double2loint(r)), a);
  const double gg = (__double2hiint(x0) >= 0) ? cs_neg(w) : w;
  *g = gg;
  *v0 = x0 - gg;
  *t = cs_rcp(s);
  // as integers: a NaN is above every number.  A zero ss makes r infinite and s
  // a NaN: tested by itself
  const long long b = __double_as_longlong(s) & 0x7fffffffffffffffll;
  return b >= least && (__double_as_longlong(ss) << 1) != 0;
}

#endif  // CS_FP64_CUH
