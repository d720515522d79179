// Shared device definitions: Cartesian index tables, compile-time loops,
// device-side records of shells / shell pairs and the Boys function.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "dd32.cuh"

namespace lgb {

// First statement of a kernel that launch_beside launches: `if (beside_block())
// return;`.  The launch after this one may start once every block of this one
// has; this one ends only after the launch before it has ended, so that an
// ordinary launch behind a group of them is behind them all.  One block more
// than the kernel asked for, the last column of the grid, waits for that (a
// wait on the way out of the working blocks cost the J/K kernels 4 to 8
// registers, 2.4 % of a 387-function chain).
__device__ __forceinline__ bool beside_block() {
  asm volatile("griddepcontrol.launch_dependents;");
  if (blockIdx.x != gridDim.x - 1) return false;
  if (blockIdx.y == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  return true;
}
// columns of working blocks
__device__ __forceinline__ unsigned besides() { return gridDim.x - 1; }

constexpr int kMaxL = 3;               // per-shell angular momentum handled by the kernels (f)
constexpr int kMaxLQuartet = 4 * kMaxL;

// ---- Cartesian components -------------------------------------------------
// Order inside a shell of angular momentum l (lowdin order, also libint2's
// default): for i = 0..l: x = l - i, for j = 0..i: y = i - j, z = j,
// i.e. xx, xy, xz, yy, yz, zz for d.  A "cumulative" index enumerates every
// component of every total 0, 1, 2, ... in that order.
__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int coff(int k) { return k * (k + 1) * (k + 2) / 6; }
__host__ __device__ constexpr int cidx(int x, int y, int z) {
  return coff(x + y + z) + (y + z) * (y + z + 1) / 2 + z;
}
__host__ __device__ constexpr int clevel(int c) {
  int k = 0;
  while (coff(k + 1) <= c) ++k;
  return k;
}
__host__ __device__ constexpr int crow(int c) {
  int r = c - coff(clevel(c)), i = 0;
  while ((i + 1) * (i + 2) / 2 <= r) ++i;
  return i;
}
__host__ __device__ constexpr int cx(int c) { return clevel(c) - crow(c); }
__host__ __device__ constexpr int cz(int c) { return c - coff(clevel(c)) - crow(c) * (crow(c) + 1) / 2; }
__host__ __device__ constexpr int cy(int c) { return clevel(c) - cx(c) - cz(c); }
__host__ __device__ constexpr int ccomp(int c, int d) { return d == 0 ? cx(c) : (d == 1 ? cy(c) : cz(c)); }
// recursion axis: first axis with a non-zero exponent
__host__ __device__ constexpr int cdir(int c) { return cx(c) > 0 ? 0 : (cy(c) > 0 ? 1 : 2); }
__host__ __device__ constexpr int cminus(int c, int d) {
  return cidx(cx(c) - (d == 0), cy(c) - (d == 1), cz(c) - (d == 2));
}
__host__ __device__ constexpr int cplus(int c, int d) {
  return cidx(cx(c) + (d == 0), cy(c) + (d == 1), cz(c) + (d == 2));
}

// compile-time loop: f(std::integral_constant<int, I>) for I in [B, E)
template <int B, int E, typename F>
__device__ __forceinline__ void sfor(F &&f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    sfor<B + 1, E>(f);
  }
}

// ---- device records ---------------------------------------------------------
// One shell pair of a species, stored in canonical order (la >= lb).  Pairs are
// grouped by class (la, lb) and, inside a class, sorted by decreasing Schwarz
// factor so that a contiguous range is one class.  R = double for the FP64
// kernels, float for the FP32 kernels (a separate copy, so the FP32 kernels
// issue no FP64 conversions).
template <typename R>
struct alignas(16) PairT {
  int sa, sb;      // shell indices inside the species
  int fa, fb;      // first basis function of each shell
  int prim0, nprim;// primitive-pair range
  int la, lb;
  R A[3];          // centre of shell a
  R AB[3];         // A - B
  R Q;             // Schwarz factor sqrt(max |(ab|ab)|) of raw integrals
  R pad;
};
using PairRec = PairT<double>;
using PairRec32 = PairT<float>;
using PairRecD = PairT<dd32>;   // double-float

// One primitive pair: exponent sum p, its reciprocal, the Gaussian-product
// centre P, P - A, and Kt = sqrt(2 pi^{5/2}) exp(-ab/p |AB|^2) c_a N_a c_b N_b / p
// (coefficients times the primitive norm of the x^l component), so that the
// quartet prefactor is Kt_ab Kt_cd / sqrt(p + q).
template <typename R>
struct alignas(16) PrimT {
  R p, inv_p, Kt, pad;
  R P[3];
  R PA[3];
};
using PrimRec = PrimT<double>;
using PrimRec32 = PrimT<float>;
// In double-float the product centre has three terms: P - Q of two pairs on
// one atom loses its leading digits, times sqrt(rho) of tight functions.
template <>
struct alignas(16) PrimT<dd32> {
  dd32 p, inv_p, Kt, pad;
  dd32 PA[3];
  float P[3][3];
  float pad2;
};
using PrimRecD = PrimT<dd32>;
template <typename R>
__device__ __forceinline__ R centre_diff(const PrimT<R> &a, const PrimT<R> &b, int d) {
  if constexpr (std::is_same<R, dd32>::value) return diff3(a.P[d], b.P[d]);
  else return a.P[d] - b.P[d];
}
template <typename R>
__device__ __forceinline__ R halved(R x) {
  if constexpr (std::is_same<R, dd32>::value) return scaled(x, 0.5f);
  else return R(0.5) * x;
}
// K x of a small whole number
template <int K, typename R>
__device__ __forceinline__ R times(R x) {
  if constexpr (K == 1) return x;
  else if constexpr (std::is_same<R, dd32>::value) return K == 2 ? scaled(x, 2.f) : x * float(K);
  else return R(K) * x;
}

constexpr double kSqrt2Pi52 = 5.914967172795612;  // sqrt(2 pi^{5/2})

// ---- Boys function ----------------------------------------------------------
// F_m(T) = int_0^1 t^{2m} exp(-T t^2) dt.
// T < kBoysTMax: Taylor series about the nearest grid point T_i = i h of a table
// of F_n(T_i) (n = 0 .. kBoysOrders-1), giving F_L, then the downward recursion
// F_m = (2T F_{m+1} + e^{-T}) / (2m+1).
// T >= kBoysTMax: F_0 = sqrt(pi/T)/2 (erfc(6) < 3e-17), upward recursion
// F_{m+1} = ((2m+1) F_m - e^{-T}) / (2T).
constexpr double kBoysH = 0.1;
constexpr double kBoysTMax = 36.0;
constexpr int kBoysPoints = 361;          // T_i = 0, 0.1, ..., 36.0
constexpr int kBoysTaylor = 9;            // terms k = 0..8 (|dT| <= 0.05: error < 6e-18)
constexpr int kBoysOrders = kMaxLQuartet + kBoysTaylor + 1;
constexpr int kBoysStride = kBoysOrders + 1;  // row i: F_0..F_{kBoysOrders-1}(T_i), then e^{-T_i}
// After that table, one table per order L = 0..kMaxLQuartet of the Taylor
// coefficients of F_L about T_i, c_k = F_{L+k}(T_i) / k! (k < kBoysTaylor),
// followed by e^{-T_i}: rows of kBoysSRow doubles, so the series is a plain
// Horner chain of FMAs in (T_i - T).
constexpr int kBoysSRow = kBoysTaylor + 1;
constexpr int kBoysScaledOff = kBoysPoints * kBoysStride;
constexpr int kBoysF64Size = kBoysScaledOff + (kMaxLQuartet + 1) * kBoysPoints * kBoysSRow;

// e^x for |x| <= h/2 = 0.05: Taylor polynomial of degree 9 (remainder below
// 0.05^10 / 10! = 2.7e-20 relative), so e^{-T} = e^{-T_i} e^{T_i - T} costs
// nine FMAs and one table read
__host__ __device__ __forceinline__ double exp_small(double x) {
  double s = 1.0 / 362880.0;  // 1/9!
  s = fma(s, x, 1.0 / 40320.0);
  s = fma(s, x, 1.0 / 5040.0);
  s = fma(s, x, 1.0 / 720.0);
  s = fma(s, x, 1.0 / 120.0);
  s = fma(s, x, 1.0 / 24.0);
  s = fma(s, x, 1.0 / 6.0);
  s = fma(s, x, 0.5);
  s = fma(s, x, 1.0);
  return fma(s, x, 1.0);
}

__device__ __forceinline__ double rsqrt_r(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_r(float x) { return rsqrtf(x); }

template <int L>
__device__ __forceinline__ void boys_f64(double T, double (&F)[L + 1], const double *__restrict__ tab) {
  if (T < kBoysTMax) {
    const int i = __double2int_rn(T * (1.0 / kBoysH));
    const double mdT = i * kBoysH - T;  // -(T - T_i)
    const double *t = tab + kBoysScaledOff + (L * kBoysPoints + i) * kBoysSRow;
    double s = __ldg(t + kBoysTaylor - 1);
#pragma unroll
    for (int k = kBoysTaylor - 1; k >= 1; --k) s = fma(s, mdT, __ldg(t + k - 1));
    F[L] = s;
    if constexpr (L > 0) {
      const double e = __ldg(t + kBoysTaylor) * exp_small(mdT);
      const double twoT = 2.0 * T;
#pragma unroll
      for (int m = L - 1; m >= 0; --m) F[m] = fma(twoT, F[m + 1], e) * (1.0 / (2 * m + 1));
    }
  } else {
    const double r = rsqrt(T);
    F[0] = 0.88622692545275801365 * r;  // sqrt(pi/T)/2
    if constexpr (L > 0) {
      // e^{-T} < 1.1e-20 above T = 46: its share of every F_m (m <= 8) there is
      // below 1e-11 relative and 1e-21 absolute, so it is left out
      const double e = T < 46.0 ? exp(-T) : 0.0;
      const double o2T = 0.5 * r * r;
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) * o2T;
    }
  }
}

// FP32 Boys function by arithmetic alone (no table reads: a warp's 32
// table rows are 32 scattered cache sectors, which bound the FP32 kernels on
// the L1 pipe while their FMA pipe idled).
//   L = 0: F_0(T) = sqrt(pi/T)/2 erf(sqrt(T)) (erff), F_0(0) = 1.
//   L > 0, T < 4: F_L(T) = e^{-T} sum_k (2T)^k / ((2L+1)(2L+3)...(2L+2k+1))
//     (a series of positive terms; kBoysSeries(L) terms leave < 1e-7 of the
//     sum at T = 4), then the downward recursion
//     F_m = (2T F_{m+1} + e^{-T}) / (2m+1).
//   L > 0, T >= 4: F_0 as above, then the upward recursion
//     F_{m+1} = ((2m+1) F_m - e^{-T}) / (2T) (stable there for m < 4).
// Relative error below 8e-7 for every m <= L <= 4 and T >= 0 (checked against
// the incomplete gamma function); FP32 evaluates only quartets whose
// contribution is bounded by the mixed-precision split.
__host__ __device__ constexpr int kBoysSeries(int L) { return L <= 1 ? 16 : (L == 2 ? 15 : 14); }
constexpr float kBoysSplitT = 4.0f;

__device__ __forceinline__ float boys0_f32(float T) {
  return T < 1e-8f ? 1.0f - T * (1.0f / 3.0f) : 0.886226925f * erff(sqrtf(T)) * rsqrtf(T);
}

template <int L>
__device__ __forceinline__ void boys_f32(float T, float (&F)[L + 1], const float *__restrict__) {
  if constexpr (L == 0) {
    F[0] = boys0_f32(T);
  } else {
    const float e = __expf(-T);
    if (T < kBoysSplitT) {
      const float twoT = 2.0f * T;
      float term = 1.0f / (2 * L + 1), sum = term;
#pragma unroll
      for (int k = 1; k <= kBoysSeries(L); ++k) {
        term *= twoT * (1.0f / (2 * L + 2 * k + 1));
        sum += term;
      }
      F[L] = e * sum;
#pragma unroll
      for (int m = L - 1; m >= 0; --m) F[m] = fmaf(twoT, F[m + 1], e) * (1.0f / (2 * m + 1));
    } else {
      F[0] = boys0_f32(T);
      const float o2T = 0.5f / T;
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = fmaf((float)(2 * m + 1), F[m], -e) * o2T;
    }
  }
}

// Boys function in double-float.  T < kBoysTMax: Taylor series of F_L about
// T_i = i / 32 (|x| <= 1/64: seven terms leave 5e-17), whose coefficients carry
// two FP32 terms up to k = 3 and one beyond (x^4 c_4 < 3e-9, so its FP32
// rounding is below 2e-16); F_{L-1}.. by the downward recursion, for L = 1 by a
// second series, which is cheaper than e^{-T}.  T >= kBoysTMax as in FP64, where
// e^{-T} (< 3e-16) is an FP32 term.
// Row i of order L (kDDRow floats): c_0..c_3 as (hi, lo), c_4, c_5, c_6, e^{-T_i} (hi, lo).
constexpr int kDDMaxL = 4;
constexpr int kDDPoints = 36 * 32 + 1;
constexpr int kDDRow = 16;
constexpr size_t kBoysDDSize = (size_t)(kDDMaxL + 1) * kDDPoints * kDDRow;

__device__ __forceinline__ dd32 boys_dd_series(const float4 &a, const float4 &b, const float4 &c, dd32 x) {
  const float t = ffma(x.hi, ffma(x.hi, c.z, c.y), c.x);
  dd32 s = fast_two_sum(b.z, ffma(x.hi, t, b.w));
  s = mad(s, x, dd32(b.x, b.y));
  s = mad(s, x, dd32(a.z, a.w));
  return mad(s, x, dd32(a.x, a.y));
}
// e^x, |x| <= 1/64
__device__ __forceinline__ dd32 exp_small_dd(dd32 x) {
  const float t = ffma(x.hi, ffma(x.hi, 1.f / 720, 1.f / 120), 1.f / 24);
  dd32 s = fast_two_sum(1.f / 6, ffma(x.hi, t, (float)(1.0 / 6 - (double)(1.f / 6))));
  s = mad(s, x, dd32(0.5f));
  s = mad(s, x, dd32(1.f));
  return mad(s, x, dd32(1.f));
}

template <int L>
__device__ __forceinline__ void boys_dd(dd32 T, dd32 (&F)[L + 1], const float *__restrict__ tab) {
  if (T.hi < (float)kBoysTMax) {
    const int i = __float2int_rn(fmul(T.hi, 32.f));
    const dd32 x = two_sum(fsub(fmul((float)i, 0.03125f), T.hi), -T.lo);
    const float4 *r = reinterpret_cast<const float4 *>(tab + ((size_t)L * kDDPoints + i) * kDDRow);
    const float4 c = __ldg(r + 2);
    F[L] = boys_dd_series(__ldg(r), __ldg(r + 1), c, x);
    if constexpr (L == 1) {
      const float4 *q = reinterpret_cast<const float4 *>(tab + (size_t)i * kDDRow);
      F[0] = boys_dd_series(__ldg(q), __ldg(q + 1), __ldg(q + 2), x);
    } else if constexpr (L > 1) {
      const dd32 e = dd32(c.w, __ldg(reinterpret_cast<const float *>(r + 3))) * exp_small_dd(x);
      const dd32 twoT = scaled(T, 2.f);
#pragma unroll
      for (int m = L - 1; m >= 0; --m) {
        const dd32 o((float)(1.0 / (2 * m + 1)), (float)(1.0 / (2 * m + 1) - (double)(float)(1.0 / (2 * m + 1))));
        F[m] = mad(twoT, F[m + 1], e);
        if (m) F[m] = F[m] * o;
      }
    }
  } else {
    const dd32 r = rsqrt_r(T);
    F[0] = r * dd32((float)0.88622692545275801365,
                    (float)(0.88622692545275801365 - (double)(float)0.88622692545275801365));
    if constexpr (L > 0) {
      const float e = __expf(-T.hi);
      const dd32 o2T = scaled(r * r, 0.5f);
#pragma unroll
      for (int m = 0; m < L; ++m) {
        dd32 v = m ? F[m] * float(2 * m + 1) : F[0];
        v.lo = fsub(v.lo, e);
        F[m + 1] = v * o2T;
      }
    }
  }
}

template <typename R>
struct BoysTab;
template <>
struct BoysTab<dd32> {
  template <int L>
  __device__ __forceinline__ static void eval(dd32 T, dd32 (&F)[L + 1], const double *, const float *tdd) {
    boys_dd<L>(T, F, tdd);
  }
};
template <>
struct BoysTab<double> {
  template <int L>
  __device__ __forceinline__ static void eval(double T, double (&F)[L + 1], const double *t64, const float *) {
    boys_f64<L>(T, F, t64);
  }
};
template <>
struct BoysTab<float> {
  template <int L>
  __device__ __forceinline__ static void eval(float T, float (&F)[L + 1], const double *, const float *t32) {
    boys_f32<L>(T, F, t32);
  }
};

}  // namespace lgb
