// pair_arith.cuh -- numbers held as the sum of two floats, and conversions between
// double, float and pairs that do not use the FP64 pipe.
//
// A warp's FP64 instruction, a conversion included, takes about 16 cycles of an SM's
// pipe here.  With cvt instructions (three for a pair) and FP64 sums the passes over the
// state of the mixed form ran at 70-80 % of that pipe and 13-26 % of the DRAM bandwidth
// (24 points at N_sh = 16); taken from the bits, the conversions run on the integer cores.
#pragma once
#include <string.h>

#ifdef __CUDACC__
#define PAIR_HD __host__ __device__ __forceinline__
#else
#define PAIR_HD inline
struct float2 { float x, y; };
#endif

namespace pnfam {

PAIR_HD unsigned long long pair_bits(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b; memcpy(&b, &x, 8); return b;
#endif
}
PAIR_HD double pair_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x; memcpy(&x, &b, 8); return x;
#endif
}
PAIR_HD unsigned pair_bits32(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  unsigned b; memcpy(&b, &x, 4); return b;
#endif
}
PAIR_HD float pair_float(unsigned b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x; memcpy(&x, &b, 4); return x;
#endif
}

// x * 2^s as a pair: the leading 24 bits, and the other 29 rounded to 24.  Exact to 2^-49
// of x for 2^-100 <= |x 2^s| < 2^127 (callers choose s so that the largest value of a
// vector is about 1), below to the least denormal float, 2^-149; overflow gives an infinity,
// as a conversion does
PAIR_HD float2 pair_split(double x, int s = 0) {
  const unsigned long long b = pair_bits(x);
  const unsigned h = (unsigned)(b >> 32), l = (unsigned)b;
  const int er = (int)((h >> 20) & 0x7ffu), e = er + s;
  const unsigned r = l & 0x1fffffffu, up = r >> 28;   // the 29 bits below the leading 24
  const unsigned m = ((h & 0xfffffu) << 3) | (l >> 29);
  const unsigned sg = h & 0x80000000u;
  float2 o;
  o.x = pair_float(sg | (((unsigned)(e - 896) << 23) + m + up));
  o.y = (float)((int)r - (int)(up << 29)) * pair_float(sg | ((unsigned)(e - 948) << 23));
  if (er == 0 || e < 949 || e > 1150) {
    o.y = 0.f;
    if (er == 2047) o.x = pair_float(sg | 0x7f800000u | (m | r ? 0x400000u : 0u));
    else if (er == 0) o.x = pair_float(sg);
    else if (e > 1150) o.x = pair_float(sg | 0x7f800000u);
    else if (e >= 872) {   // the scale of the low part, or of both, in two steps
      const float q = 7.888609052210118e-31f;   // 2^-100
      if (e < 897) o.x = pair_float(sg | ((127u << 23) + m + up)) * pair_float((unsigned)(e - 796) << 23) * q;
      else o.y = (float)((int)r - (int)(up << 29)) * pair_float(sg | ((unsigned)(e - 848) << 23)) * q;
    } else o.x = pair_float(sg);
  }
  return o;
}

// (float)x, rounded to nearest even
PAIR_HD float f32_of(double x) {
  const unsigned long long b = pair_bits(x);
  const unsigned h = (unsigned)(b >> 32), l = (unsigned)b, sg = h & 0x80000000u;
  const int e = (int)((h >> 20) & 0x7ffu);
  const unsigned m = ((h & 0xfffffu) << 3) | (l >> 29), r = l & 0x1fffffffu;
  const unsigned up = (r > 0x10000000u || (r == 0x10000000u && (m & 1u))) ? 1u : 0u;
  unsigned o = sg | (((unsigned)(e - 896) << 23) + m + up);
  if (e < 897 || e > 1150) {
    if (e == 2047) o = sg | 0x7f800000u | (m | r ? 0x400000u : 0u);
    else if (e > 1150) o = sg | 0x7f800000u;
    else if (e < 872) o = sg;   // below half of the least denormal
    else {                      // a denormal float: multiples of 2^-149
      const unsigned long long q = (b & 0xfffffffffffffULL) | 0x10000000000000ULL;
      const int n = 926 - e;    // bits dropped, 30 ... 54
      const unsigned long long k = q >> n, d = q & ((1ULL << n) - 1), half = 1ULL << (n - 1);
      o = sg | (unsigned)(k + ((d > half || (d == half && (k & 1))) ? 1 : 0));
    }
  }
  return pair_float(o);
}

// (double)x * 2^s; results below the normal range are 0
PAIR_HD double f64_of(float x, int s = 0) {
  const unsigned b = pair_bits32(x);
  unsigned m = b & 0x7fffffu;
  int e = (int)((b >> 23) & 0xffu);
  const unsigned long long sg = (unsigned long long)(b & 0x80000000u) << 32;
  if (e == 0 && m) {   // a denormal: normalise
    e = 1;
    do { m <<= 1; --e; } while (!(m & 0x800000u));
    m &= 0x7fffffu;
    e += 896 + s;
  } else if (e == 0) {
    return pair_double(sg);
  } else {
    e = e == 255 ? 2047 : e + 896 + s;
  }
  if (e <= 0) return pair_double(sg);
  if (e >= 2047) return pair_double(sg | 0x7ff0000000000000ULL | (((b >> 23) & 0xffu) == 255 ? (unsigned long long)m << 29 : 0));
  return pair_double(sg | ((unsigned long long)e << 52) | ((unsigned long long)m << 29));
}

// s for which m * 2^s lies in [1, 2), m >= 0; 0 for 0, denormals, infinity and NaN
PAIR_HD int pair_scale(double m) {
  const int e = (int)((pair_bits(m) >> 52) & 0x7ffu);
  if (e == 0 || e == 2047) return 0;
  const int s = 1023 - e;
  return s > 900 ? 900 : s < -900 ? -900 : s;
}

// the larger of two non-negative doubles given by their bits, which order like them; a
// NaN is passed over, as fmax does
PAIR_HD unsigned long long abs_max(unsigned long long m, double x) {
  const unsigned long long b = pair_bits(x) & 0x7fffffffffffffffULL;
  return b > m && b <= 0x7ff0000000000000ULL ? b : m;
}

#ifdef __CUDACC__
// s += a*b: the exact error of the leading product (by FMA, after Dekker's product) and the
// cross terms go to the low part, the leading sum is Knuth's two-sum (rounded operations that
// the compiler may not contract)
__device__ __forceinline__ void pair_fma(float2& s, float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = fmaf(a.x, b.x, -p);
  e = fmaf(a.x, b.y, e);
  e = fmaf(a.y, b.x, e);
  const float t = __fadd_rn(s.x, p);
  const float z = __fsub_rn(t, s.x);
  const float err = __fadd_rn(__fsub_rn(s.x, __fsub_rn(t, z)), __fsub_rn(p, z));
  s.x = t;
  s.y = __fadd_rn(s.y, __fadd_rn(err, e));
}
__device__ __forceinline__ double pair_value(float2 a, int s = 0) { return f64_of(a.x, s) + f64_of(a.y, s); }
// the warp's sums of a (lanes 0 ... 15) and of b (lanes 16 ... 31), in FP64: as pairs across
// the lanes they were 1.2 to 1.8 times as far from the exact sums (32 products of a lane,
// measured over 20,000 of them). The halves of the warp take a sum each, so that the two
// cost 7 FP64 instructions and not 12
__device__ __forceinline__ double pair_warp_sums(float2 a, float2 b, int lane) {
  const double x = pair_value(a), y = pair_value(b);
  double r = (lane & 16 ? y : x) + __shfl_xor_sync(0xffffffffu, lane & 16 ? x : y, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}
// the largest of a warp's bit patterns
__device__ __forceinline__ unsigned long long warp_abs_max(unsigned long long m) {
  const unsigned h = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32));
  const unsigned l = __reduce_max_sync(0xffffffffu, (unsigned)(m >> 32) == h ? (unsigned)m : 0u);
  return ((unsigned long long)h << 32) | l;
}
#endif

}  // namespace pnfam
