// Double-float arithmetic: a value is the unevaluated sum of two FP32 numbers,
// about 47 significant bits.  GB300 issues one FP64 instruction where it issues
// 63 FP32 instructions; the products and sums below (Dekker's product error by
// fused multiply-add, Knuth's two-sum) take 4 to 16 FP32 instructions each.
// The pairs are not renormalised after each operation (pair arithmetic, Lange
// and Rump 2020): lo may exceed half an ulp of hi, and after a cancellation even
// hi itself, but the error of a result stays within some 2^-46 of the
// magnitudes it was computed from, which is how FP64 rounding behaves too.  Used
// where such an error lies below the FP64 rounding of the sums it goes into.
#pragma once
#include <cuda_runtime.h>

namespace lgb {

struct dd32 {
  float hi, lo;
  dd32() = default;
  __host__ __device__ __forceinline__ explicit constexpr dd32(float h, float l = 0.f) : hi(h), lo(l) {}
};

// Every operation is an explicitly rounded one, so the compiler can neither
// contract nor reorder it.
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fadd_rn(a, -b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// a + b with |a| >= |b|
__device__ __forceinline__ dd32 fast_two_sum(float a, float b) {
  const float s = fadd(a, b);
  return dd32(s, fsub(b, fsub(s, a)));
}
__device__ __forceinline__ dd32 two_sum(float a, float b) {
  const float s = fadd(a, b), bb = fsub(s, a);
  return dd32(s, fadd(fsub(a, fsub(s, bb)), fsub(b, bb)));
}
__device__ __forceinline__ dd32 operator-(dd32 a) { return dd32(-a.hi, -a.lo); }
__device__ __forceinline__ dd32 operator+(dd32 a, dd32 b) {
  const dd32 s = two_sum(a.hi, b.hi);
  return dd32(s.hi, fadd(s.lo, fadd(a.lo, b.lo)));
}
__device__ __forceinline__ dd32 operator-(dd32 a, dd32 b) { return a + (-b); }
__device__ __forceinline__ dd32 operator*(dd32 a, dd32 b) {
  const float p = fmul(a.hi, b.hi);
  return dd32(p, ffma(a.lo, b.hi, ffma(a.hi, b.lo, ffma(a.hi, b.hi, -p))));
}
__device__ __forceinline__ dd32 operator*(dd32 a, float b) {
  const float p = fmul(a.hi, b);
  return dd32(p, ffma(a.lo, b, ffma(a.hi, b, -p)));
}
__device__ __forceinline__ dd32 &operator+=(dd32 &a, dd32 b) { return a = a + b; }
// times a power of two
__device__ __forceinline__ dd32 scaled(dd32 a, float f) { return dd32(fmul(a.hi, f), fmul(a.lo, f)); }

// a b + c and a b + c d; the FP64 and FP32 kernels use the same names
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ dd32 mad(dd32 a, dd32 b, dd32 c) {
  const float p = fmul(a.hi, b.hi);
  const dd32 s = two_sum(p, c.hi);
  const float e = ffma(a.lo, b.hi, ffma(a.hi, b.lo, ffma(a.hi, b.hi, -p)));
  return dd32(s.hi, fadd(s.lo, fadd(e, c.lo)));
}
__device__ __forceinline__ double mad2(double a, double b, double c, double d) { return fma(a, b, c * d); }
__device__ __forceinline__ float mad2(float a, float b, float c, float d) { return fmaf(a, b, c * d); }
__device__ __forceinline__ dd32 mad2(dd32 a, dd32 b, dd32 c, dd32 d) {
  const float p = fmul(a.hi, b.hi), q = fmul(c.hi, d.hi);
  const dd32 s = two_sum(p, q);
  const float e = ffma(a.lo, b.hi, ffma(a.hi, b.lo, ffma(a.hi, b.hi, -p)));
  const float f = ffma(c.lo, d.hi, ffma(c.hi, d.lo, ffma(c.hi, d.hi, -q)));
  return dd32(s.hi, fadd(s.lo, fadd(e, f)));
}

// 1 / sqrt(a): y = rsqrtf(a), r = 1 - a y^2 evaluated exactly to ~2^-48, then
// y (1 + r / 2 + 3 r^2 / 8) (the binomial series of (1 - r)^(-1/2))
__device__ __forceinline__ dd32 rsqrt_r(dd32 a) {
  const float y = rsqrtf(a.hi);
  const float p = fmul(y, y), pe = ffma(y, y, -p);
  const float u = fmul(a.hi, p);
  const float ue = ffma(a.lo, p, ffma(a.hi, pe, ffma(a.hi, p, -u)));
  const float r = fsub(fsub(1.f, u), ue);
  return fast_two_sum(y, fmul(y, ffma(fmul(0.375f, r), r, fmul(0.5f, r))));
}

// a0 + a1 + a2 - (b0 + b1 + b2) of two three-term expansions: the difference
// of two coordinates that agree in their leading digits keeps 48 of its own
__device__ __forceinline__ dd32 diff3(const float (&a)[3], const float (&b)[3]) {
  const dd32 d0 = two_sum(a[0], -b[0]), d1 = two_sum(a[1], -b[1]);
  const dd32 m = two_sum(d0.lo, d1.hi);
  const dd32 h = two_sum(d0.hi, m.hi);
  return dd32(h.hi, fadd(h.lo, fadd(m.lo, fadd(d1.lo, fsub(a[2], b[2])))));
}

// The FP64 number nearest to hi + lo, by integer instructions alone (a
// conversion costs as much as an FP64 operation).  |hi| below 2^-100 gives
// hi alone; zero, infinities and NaN of hi are kept.
__device__ __forceinline__ double to_double(dd32 v) {
  const dd32 a = two_sum(v.hi, v.lo);
  const int h = __float_as_int(a.hi), e = (h >> 23) & 255;
  if (e == 0) return 0.0;
  const long long sign = (long long)(h & 0x80000000) << 32;
  if (e == 255) return __longlong_as_double(sign | 0x7ff0000000000000ll | ((long long)(h & 0x7fffff) << 29));
  long long m = ((long long)(e + 896) << 52) | ((long long)(h & 0x7fffff) << 29);
  if (e > 27) {
    // lo in units of the last place of the FP64 number: below 2^29 + rounding
    float l = h < 0 ? -a.lo : a.lo;
    l = fmul(fmul(l, __int_as_float((254 - e) << 23)), 0x1p52f);   // 2^(127 - e) 2^52
    // just above a power of two the places below are half as wide
    if ((h & 0x7fffff) == 0 && l < 0.f) l = fadd(l, l);
    m += __float2int_rn(l);
  }
  return __longlong_as_double(sign | m);
}

// hi + lo of a double (host)
inline dd32 split_double(double d) {
  const float h = (float)d;
  return dd32(h, (float)(d - (double)h));
}

}  // namespace lgb
