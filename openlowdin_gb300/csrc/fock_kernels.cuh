// Kernel templates: Schwarz factors, intra-species J/K, fused inter-species
// coupling and first-quarter transforms.  Included by the translation units
// that instantiate them for a set of quartet classes.
#pragma once
#include <type_traits>

#include "eri.cuh"
#include "kernels.cuh"

namespace lgb {

template <typename R>
__device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += shfl_xor(v, o);
  return v;
}

// The FP64 pipe of this GPU issues at 1/64 of the FP32 rate, so comparisons
// and maxima of non-negative doubles are done on their bit patterns (IEEE
// order of non-negative values = unsigned integer order of their bits):
// integer instructions, identical decisions.
__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ unsigned abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
// |v| < t and |v| > t for a non-negative threshold t
template <typename R>
__device__ __forceinline__ bool abs_below(R v, R t) { return abs_bits(v) < abs_bits(t); }
template <typename R>
__device__ __forceinline__ bool abs_above(R v, R t) { return abs_bits(v) > abs_bits(t); }
// 2^k, k = 0..3 (quartet degeneracies), from the exponent field alone
template <typename R>
__device__ __forceinline__ auto pow2(int k) {
  if constexpr (std::is_same<R, double>::value) return __longlong_as_double((long long)(1023 + k) << 52);
  else return __int_as_float((127 + k) << 23);
}

// largest shell-block maximum |D| over the six index pairs of a quartet, by bit
// patterns: the norms are >= 0, and a NaN orders above every number, so that no
// quartet that meets one is screened
template <typename T>
__device__ __forceinline__ T dnorm6(const T *__restrict__ Dn, int nsh, int a, int b, int c, int d) {
  using U = std::conditional_t<std::is_same<T, double>::value, unsigned long long, unsigned>;
  const U *u = reinterpret_cast<const U *>(Dn);
  U m = __ldg(u + a * nsh + b);
  m = max(m, __ldg(u + a * nsh + c));
  m = max(m, __ldg(u + b * nsh + c));
  m = max(m, __ldg(u + a * nsh + d));
  m = max(m, __ldg(u + b * nsh + d));
  m = max(m, __ldg(u + c * nsh + d));
  if constexpr (std::is_same<T, double>::value) return __longlong_as_double((long long)m);
  else return __uint_as_float(m);
}

// Per-system build flag of a batch (LowdinGB300_batch_set_active): off
// (converged, nothing built), on, or held in FP64 (mixed builds evaluate all
// of the system's quartets in their FP64 launches).  Tasks without a flag are on.
constexpr int kSysOff = 0, kSysOn = 1, kSysFP64 = 2;
__device__ __forceinline__ int system_flag(const int *f) { return f ? __ldg(f) : kSysOn; }

// task owning flattened block b: last task with blk0 <= b (tasks sorted by blk0)
template <typename T>
__device__ __forceinline__ int find_task(const T *__restrict__ tasks, int ntasks, int b) {
  int lo = 0, hi = ntasks - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&tasks[mid].blk0) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ double scaled(double a, double f) { return a * f; }
__device__ __forceinline__ float scaled(float a, float f) { return a * f; }

template <typename R>
__device__ __forceinline__ void atomic_acc(double *g64, float *g32, size_t i, R v) {
  if constexpr (std::is_same<R, double>::value) atomicAdd(g64 + i, v);
  else if constexpr (std::is_same<R, dd32>::value) atomicAdd(g64 + i, to_double(v));
  else atomicAdd(g32 + i, v);
}

// |v| > cut of a raw integral
__device__ __forceinline__ bool above_cut(double v, double cut) { return abs_above(v, cut); }
__device__ __forceinline__ bool above_cut(dd32 v, double cut) {
  const float a = fabsf(fadd(v.hi, v.lo)), c = (float)cut;
  if (fabsf(a - c) <= 1e-5f * c) return abs_above(to_double(v), cut);   // too near for FP32
  return !(a <= c);   // NaN is kept, as abs_above keeps it
}

// element i of a matrix kept in FP64, FP32 and double-float
template <typename R>
__device__ __forceinline__ R elem(const double *m64, const float *m32, const float2 *md, int i) {
  if constexpr (std::is_same<R, double>::value) return __ldg(m64 + i);
  else if constexpr (std::is_same<R, dd32>::value) {
    const float2 v = __ldg(md + i);
    return dd32(v.x, v.y);
  } else return __ldg(m32 + i);
}

// FP32 Schwarz factor of a record of any precision (that of its FP32 copy)
__device__ __forceinline__ float schwarz32(const PairRec &p) { return (float)p.Q; }
__device__ __forceinline__ float schwarz32(const PairRec32 &p) { return p.Q; }
__device__ __forceinline__ float schwarz32(const PairRecD &p) { return p.Q.hi; }

// Bound of the double-float quartets of a species: `tier` (kTierBound times
// its largest product of Schwarz factors) times the largest density element,
// and `cap` at most.  Zero, so that everything stays in FP64, for densities
// whose products could leave the FP32 exponent range, infinities and NaN.
__device__ __forceinline__ float tier_bound(float tier, float d, float cap) {
  return d > 1e-12f && d < 1e20f ? fminf(tier * d, cap) : 0.f;
}

// ----------------------------------------------------------------- Schwarz --
template <int LA, int LB>
__global__ void __launch_bounds__(128) schwarz_kernel(SchwarzParams P) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P.np) return;
  const PairRec pr = P.pairs[P.p0 + t];
  constexpr int N = ncart(LA) * ncart(LB);
  double I[N * N];
  eri_quartet<double, LA, LB, LA, LB>(pr, P.prims + pr.prim0, pr, P.prims + pr.prim0, P.boys.f64, P.boys.dd, I);
  double m = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) m = fmax(m, fabs(I[i * N + i]));
  P.Q[P.p0 + t] = sqrt(m);
}

// The six updates of one quartet: g34 += D12 v, the exchange ones g13, g14,
// g24, g23 += hdeg D v go to the FP64 (or FP32) accumulator, g12 += D34 v to the
// caller's bra-block sums.
template <typename R, int LA, int LB, int LC, int LD, typename DF, typename S>
__device__ __forceinline__ void jk_digest(const R (&I)[QClass<LA, LB, LC, LD>::NINT], const DF &D, int n, int fa,
                                          int fb, int fc, int fd, S deg, R hdeg, double *G, float *G32,
                                          R (&j12)[ncart(LA) * ncart(LB)]) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  // density blocks of the quartet, all asked for at once: one at a time behind
  // the atomics before them they would cost a trip to L2 each
  R dcd[NC][ND], dac[NA][NC], dad[NA][ND], dbc[NB][NC], dbd[NB][ND];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int d = 0; d < ND; ++d) dcd[c][d] = D((fc + c) * n + fd + d);
#pragma unroll
  for (int a = 0; a < NA; ++a) {
#pragma unroll
    for (int c = 0; c < NC; ++c) dac[a][c] = D((fa + a) * n + fc + c);
#pragma unroll
    for (int d = 0; d < ND; ++d) dad[a][d] = D((fa + a) * n + fd + d);
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int c = 0; c < NC; ++c) dbc[b][c] = D((fb + b) * n + fc + c);
#pragma unroll
    for (int d = 0; d < ND; ++d) dbd[b][d] = D((fb + b) * n + fd + d);
  }
  auto Iat = [&](int a, int b, int c, int d) -> R { return I[((a * NB + b) * NC + c) * ND + d]; };
  // J12: bra block, summed over this block's kets; J34
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const R w = scaled(dcd[c][d], deg);
      R s = R(0);
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          j12[a * NB + b] = mad(w, Iat(a, b, c, d), j12[a * NB + b]);
          s = mad(D((fa + a) * n + fb + b), Iat(a, b, c, d), s);
        }
      atomic_acc<R>(G, G32, (size_t)(fc + c) * n + fd + d, scaled(s, deg));
    }
  // K13 (i,k) += D(j,l), K14 (i,l) += D(j,k)
#pragma unroll
  for (int a = 0; a < NA; ++a) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      R s = R(0);
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int d = 0; d < ND; ++d) s = mad(dbd[b][d], Iat(a, b, c, d), s);
      atomic_acc<R>(G, G32, (size_t)(fa + a) * n + fc + c, s * hdeg);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      R s = R(0);
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int c = 0; c < NC; ++c) s = mad(dbc[b][c], Iat(a, b, c, d), s);
      atomic_acc<R>(G, G32, (size_t)(fa + a) * n + fd + d, s * hdeg);
    }
  }
  // K24 (j,l) += D(i,k), K23 (j,k) += D(i,l)
#pragma unroll
  for (int b = 0; b < NB; ++b) {
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      R s = R(0);
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) s = mad(dac[a][c], Iat(a, b, c, d), s);
      atomic_acc<R>(G, G32, (size_t)(fb + b) * n + fd + d, s * hdeg);
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      R s = R(0);
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int d = 0; d < ND; ++d) s = mad(dad[a][d], Iat(a, b, c, d), s);
      atomic_acc<R>(G, G32, (size_t)(fb + b) * n + fc + c, s * hdeg);
    }
  }
}

// --------------------------------------------------------------------- J/K --
// Warp y of a block takes bra pair tile_y * bras + y of its task and the ket
// pairs tile_x * kets + (lane mod kets): one quartet per lane, or, for
// contracted classes (kets < 32), 32 / kets lanes per quartet, of which the
// first digests it.  The 32 lanes of a warp share the bra pair, so the
// bra-block Coulomb term is reduced across the warp before its atomics.
// Digestion follows the six updates of a permutation-unique quartet
// (g12 += D34 v, g34 += D12 v, g13/g24/g14/g23 += 0.5 f D v, all x degeneracy);
// with G = (Gacc + Gacc^T)/4 this is J[D] + f K[D].
// Screening bound: plain launches (split = 0) use the FP64 product
// Q_ab Q_cd max|D| as the reference does; mixed launches compute it in FP32
// from the FP32 records in both kernels, so each quartet lands in exactly one
// of the FP64 (bound >= split) and FP32 (bound < split) launches.
// Tier: the FP64 and the double-float launch of a class compute the same FP32
// bound and divide the quartets at tier_bound; the screening decision itself is
// the FP64 one in both (taken from FP32 only where that cannot differ).
// Blocks per SM the registers are cut for.  The light double-float classes wait
// on loads (L1 hits half of the scattered density and norm reads), so more warps
// pay until spills outweigh them: 387-function chain, (ps|ss) 5.5 ms at 4
// blocks, 4.6 at 5, 5.3 at 6; (ss|ss) 2.2 -> 1.85 at 8; (ps|ps) 3.8 -> 3.6 and
// (pp|ss) 2.1 -> 1.6 at 4.  FP64 and FP32: where one block is enough, the compiler
// takes 1.6 to 2.5 times the registers that it did without a number.  FP64 alone
// (the allocation-free entry), one block -> these: 156-function chain 2.50 -> 2.35
// ms, 4 waters 0.87 -> 0.82, 387-function chain 39.9 -> 38.4; with more blocks
// ((ss|ss) 8, (ps|ss) 6, (ps|ps) 5, (pp|ps) 3) 2.31, 0.81 and 37.9, but contracted
// waters 2.5 -> 2.7.  FP32 (bra rows off), a mixed batch of 32 chains 38.4 -> 35.9.
template <typename R, int LA, int LB, int LC, int LD>
constexpr int jk_min_blocks() {
  constexpr int N = QClass<LA, LB, LC, LD>::NINT;
  if (std::is_same<R, double>::value) return N == 1 ? 6 : N <= 3 ? 4 : N <= 9 ? 3 : N <= 27 ? 2 : 1;
  if (std::is_same<R, float>::value) return N == 1 ? 10 : N <= 9 ? 8 : N <= 27 ? 5 : N <= 81 ? 3 : 1;
  return N == 1 ? 8 : N <= 3 ? 5 : N <= 9 ? 4 : 1;
}
template <typename R, int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128, jk_min_blocks<R, LA, LB, LC, LD>()) jk_tasks_kernel(const JKTask *__restrict__ tasks, TaskLaunch TL) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr bool F64 = std::is_same<R, double>::value, DD = std::is_same<R, dd32>::value;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  // The tile's ket pairs (shared by its bra warps) and the first primitive
  // pair of each, staged in shared memory by coalesced 16-byte copies.
  // Strides 80 / 112 B (pairs) and 48 / 80 / 96 B (primitives) keep the per-lane
  // 16-byte reads nearly free of bank conflicts.
  struct alignas(16) SPair {
    PairT<R> p;
    int4 pad;
  };
  __shared__ SPair sk[32];
  __shared__ PrimT<R> skp[32];
  const int slices = TL.tile.slices;
  int blk = blockIdx.x, slice = 0;
  if (slices > 1) {
    blk = blockIdx.x / slices;
    slice = blockIdx.x - blk * slices;
  }
  const int t = find_task(tasks, TL.ntasks, blk);
  const JKTask &T = tasks[t];
  const int act = system_flag(T.active);
  if (act == kSysOff) return;   // converged system: nothing to build
  const bool all64 = act == kSysFP64;   // system held in FP64: the launches above the split take it all
  if (all64 && TL.mixed && TL.lower) return;
  const int local = blk - T.blk0;
  const int kets = TL.tile.kets, parts = 32 / kets, bras = blockDim.y;
  const int ty = local / T.nbx, b0 = ty * bras;
  int k0 = (local - ty * T.nbx) * TL.tile.chunk * kets;
  int kend = min(T.nket, k0 + TL.tile.chunk * kets);
  if (T.triangle) kend = min(kend, b0 + bras);
  if (k0 >= kend) return;
  // The quartets of this launch have lo <= b (b < split in the FP32 half), b the
  // FP32 bound: Q_ab Q_cd times, for screened species, the largest of the six
  // shell-block norms,
  float lo = 0.f;
  if (TL.mixed) {
    const float cutoff = T.screen ? fmaxf(TL.eps32, all64 ? 0.f : TL.skip) : 0.f;
    lo = TL.lower || all64 ? cutoff : fmaxf(cutoff, TL.split32);
  }
  // and, w being that bound (for species without screening, Q_ab Q_cd times the
  // largest norm of all), w >= tb in the FP64 launch, w < tb in the
  // double-float one
  const float dmax = T.Dnmax32 ? __ldg(T.Dnmax32) : -1.f;
  float tb = TL.tier == Tier::all ? 0.f : tier_bound(T.tier, dmax, kTierCap);
  if (TL.tier != Tier::all && TL.mixed && !all64) tb = fmaxf(tb, tier_bound(kMixedTier * T.tier, dmax, TL.tier_cap));
  if (TL.tier == Tier::lower && (tb == 0.f || (T.screen && !(lo < tb)))) return;
  // Pairs are sorted by decreasing Schwarz factor inside a class and Dnmax32
  // bounds the six norms, so the first bra and the first ket of a range bound
  // every quartet after them (FP32 rounding is monotonic, same order of
  // products; plain builds screen in FP64, with room for that rounding): the
  // block leaves, before staging records, a range that cannot reach lo.
  const float qb0 = T.pairs32[T.bra0 + b0].Q;
  const float reach = TL.mixed ? lo : (T.screen ? TL.eps32 * 0.99999f : 0.f);
  const float tier_reach = TL.tier == Tier::upper ? tb : 0.f;
  auto out_of_reach = [&](int k) {
    const float qq = qb0 * T.pairs32[T.ket0 + k].Q;
    if (T.screen) return dmax >= 0.f && qq * dmax < fmaxf(reach, tier_reach);
    return qq < reach || (TL.tier == Tier::upper && qq * dmax < tier_reach);
  };
  if (out_of_reach(k0)) return;
  const PairT<R> *pairs;
  const PrimT<R> *prims;
  if constexpr (F64) {
    pairs = T.pairs; prims = T.prims;
  } else if constexpr (DD) {
    pairs = T.pairsd; prims = T.primsd;
  } else {
    pairs = T.pairs32; prims = T.prims32;
  }
  auto D = [&](int i) { return elem<R>(T.Ds, T.Ds32, T.Dd, i); };
  const int n = T.n;
  double *G = T.Gacc;
  float *G32 = T.Gacc32;
  const int kl = threadIdx.x & (kets - 1), part = parts == 1 ? 0 : threadIdx.x / kets;
  const int bpos = b0 + threadIdx.y;
  const int bi = T.bra0 + min(bpos, T.nbra - 1);
  const PairT<R> &bra = pairs[bi];
  const int fa = bra.fa, fb = bra.fb;
  const float qbra = T.pairs32[bi].Q;
  R hf;
  if constexpr (F64) hf = T.hf;
  else if constexpr (DD) hf = dd32(T.hfd.x, T.hfd.y);
  else hf = T.hf32;
  R j12[NA * NB];
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) j12[x] = R(0);
  unsigned cnt = 0;
  bool worked = false;
  for (bool first = true; k0 < kend; k0 += kets, first = false) {
    if (!first && out_of_reach(k0)) break;   // every later ket is out of reach too
    __syncwarp();
    __syncthreads();                         // the previous tile has been read
    {
      constexpr int WP = sizeof(PairT<R>) / 16, WQ = sizeof(PrimT<R>) / 16;
      const int tid = threadIdx.y * 32 + threadIdx.x;
      for (int w = tid; w < kets * WP; w += 32 * bras) {
        const int r = w / WP, k = w % WP;
        const int kr = T.ket0 + min(k0 + r, T.nket - 1);
        reinterpret_cast<int4 *>(&sk[r].p)[k] = __ldg(reinterpret_cast<const int4 *>(pairs + kr) + k);
      }
      __syncthreads();
      for (int w = tid; w < kets * WQ; w += 32 * bras) {
        const int r = w / WQ, k = w % WQ;
        reinterpret_cast<int4 *>(skp + r)[k] = __ldg(reinterpret_cast<const int4 *>(prims + sk[r].p.prim0) + k);
      }
      __syncthreads();
    }
    const int kpos = k0 + kl;
    if (bpos >= T.nbra) continue;  // warp-uniform
    bool active = kpos < T.nket && (!T.triangle || kpos <= bpos);
    const int ki = T.ket0 + min(kpos, T.nket - 1);
    const PairT<R> &ket = sk[kl].p;
    if (TL.mixed || TL.tier != Tier::all) {
      // FP32 bound from the FP32 Schwarz factors and norms, identical in every
      // launch of the class
      float b = qbra * schwarz32(ket);
      const float qq = b;
      if (T.screen) b *= dnorm6(T.Dn32, T.nsh, bra.sa, bra.sb, ket.sa, ket.sb);
      const float w = T.screen ? b : qq * dmax;
      if (TL.mixed) {
        if (T.screen && b < fmaxf(TL.eps32, all64 ? 0.f : TL.skip)) active = false;   // no skip in an FP64 check
        if (!all64 && (TL.lower ? !(b < TL.split32) : (b < TL.split32))) active = false;
      } else if (T.screen && b < 1.00001f * TL.eps32) {
        if (b < 0.99999f * TL.eps32) active = false;
        else if (active) {
          // too near the threshold for FP32 to decide
          const double b64 = T.pairs[bi].Q * T.pairs[ki].Q * dnorm6(T.Dn, T.nsh, bra.sa, bra.sb, ket.sa, ket.sb);
          if (abs_below(b64, TL.eps)) active = false;
        }
      }
      if (TL.tier != Tier::all) {
        if (TL.tier == Tier::upper ? w < tb : !(w < tb)) active = false;
      }
    } else if (T.screen) {
      double qk;
      if constexpr (F64) qk = ket.Q;
      else qk = T.pairs[ki].Q;
      const double b = T.pairs[bi].Q * qk * dnorm6(T.Dn, T.nsh, bra.sa, bra.sb, ket.sa, ket.sb);
      if (abs_below(b, TL.eps)) active = false;
    }
    const unsigned live = __ballot_sync(0xffffffffu, active && part == 0);
    if (!__any_sync(0xffffffffu, active)) continue;
    if (slice == 0) cnt += __popc(live);
    else {   // quartets without a primitive quartet in this slice
      if (slice * parts >= bra.nprim * ket.nprim) active = false;
      if (!__any_sync(0xffffffffu, active)) continue;
    }
    worked = true;
    R I[Q::NINT];
    if (active || parts > 1) {
      const PrimT<R> *kp = ket.nprim == 1 ? skp + kl : prims + ket.prim0;
      eri_quartet<R, LA, LB, LC, LD>(bra, prims + bra.prim0, ket, kp, TL.boys.f64, TL.boys.dd, I, part, parts, active,
                                     slice, slices);
      if (part) active = false;   // the quartet is digested by its first lane
    }
    if (!active) continue;   // no warp-wide step follows inside the loop
    const auto deg = pow2<R>((bra.sa != bra.sb) + (ket.sa != ket.sb) + (bi != ki));
    jk_digest<R, LA, LB, LC, LD>(I, D, n, fa, fb, ket.fa, ket.fb, deg, scaled(hf, deg), G, G32, j12);
  }
  if (!worked) return;   // warp-uniform
  __syncwarp();
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) {
    const R v = warp_sum(j12[x]);
    if (threadIdx.x == 0) atomic_acc<R>(G, G32, (size_t)(fa + x / NB) * n + fb + x % NB, v);
  }
  if (T.count && cnt && threadIdx.x == 0) atomicAdd(T.count, (unsigned long long)cnt);
}

// ------------------------------------------------------- J/K, FP32 bra rows --
// FP32 half of a mixed J/K build, one block per bra pair (a b| of a task; its
// kRowWarps warps take the task's ket pairs 32 at a time).  The exchange
// updates of a quartet touch only rows fa.. and fb.. of the output (K13, K14
// on the rows of shell a, K23, K24 on those of shell b) and read only those
// rows of D, so the block keeps both in shared memory, interleaved by column
// (Drow[col][r], Krow[col][r], r < NA + NB, padded to an odd pitch so that
// random columns spread over the banks), together with the largest
// shell-block norm of shells a and b against every shell (Dnab[s] =
// max(|D|_{a s}, |D|_{b s})), which gives four of the six screening norms in
// two reads.  The ket side is read from pair-indexed arrays when the build
// provides them (JKTask::Dp32 / DnP32 / Jp32: per ket pair its D block, its
// shell-block norm and its Coulomb accumulator, element-major inside the ket
// class, so a warp's 32 kets are one coalesced line per element), else from
// the n x n matrices.  The bra Coulomb block (J12) is summed in registers
// over every ket of the warp before one warp reduction.  At the end the
// exchange rows go to the global accumulator (non-zero entries only).
// Quartet selection, bound and arithmetic are those of jk_tasks_kernel's FP32
// launch (same FP32 bound, same screening and split), so the quartets taken
// and the integrals are the same; only the order of the FP32 additions differs.
template <typename T>
__device__ __forceinline__ int find_task_rows(const T *__restrict__ tasks, int ntasks, int b) {
  int lo = 0, hi = ntasks - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&tasks[mid].rblk0) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(32 * kRowWarps) jk32_row_kernel(const JKTask *__restrict__ tasks, TaskLaunch TL) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND, NR = NA + NB, NRP = row_pitch(NA + NB);
  extern __shared__ float rsm[];
  const int t = find_task_rows(tasks, TL.ntasks, blockIdx.x);
  const JKTask &T = tasks[t];
  if (system_flag(T.active) != kSysOn) return;   // converged, or held in FP64
  const int bpos = blockIdx.x - T.rblk0;
  if (bpos >= T.nbra) return;
  const int bi = T.bra0 + bpos;
  const int nk = T.triangle ? bpos + 1 : T.nket;  // ket positions [0, nk)
  const int n = T.n, nsh = T.nsh;
  const PairRec32 bra = T.pairs32[bi];
  const PrimRec32 *__restrict__ prims = T.prims32;
  const float cutoff = fmaxf(TL.eps32, TL.skip);
  // kets are sorted by decreasing Schwarz factor: bra.Q Q(ket k0) Dnmax32 bounds
  // every quartet bound from ket position k0 on (same FP32 product order)
  const float dmax = (T.screen && T.Dnmax32) ? __ldg(T.Dnmax32) : -1.f;
  auto below_from = [&](int k0) {
    const float qk = T.soa32 ? T.soa32[kSoaQ * T.npairs + T.ket0 + k0] : T.pairs32[T.ket0 + k0].Q;
    return dmax >= 0.f && bra.Q * qk * dmax < cutoff;
  };
  if (below_from(0)) return;   // nothing of this bra row reaches the cutoff
  float *Drow = rsm;                 // [n][NRP]: D(fa + r, col) for r < NA, D(fb + r - NA, col) after
  float *Krow = rsm + NRP * n;       // [n][NRP]: exchange accumulators of the same rows
  float *Dnab = Krow + NRP * n;      // [nsh]
  for (int i = threadIdx.x; i < NRP * n; i += blockDim.x) {
    const int c = i / NRP, r = i - c * NRP;
    float v = 0.f;
    if (r < NR) v = __ldg(T.Ds32 + (size_t)(r < NA ? bra.fa + r : bra.fb + (r - NA)) * n + c);
    Drow[i] = v;
    Krow[i] = 0.f;
  }
  if (T.screen)
    for (int i = threadIdx.x; i < nsh; i += blockDim.x)
      Dnab[i] = fmaxf(__ldg(T.Dn32 + (size_t)bra.sa * nsh + i), __ldg(T.Dn32 + (size_t)bra.sb * nsh + i));
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float hf = T.hf32;
  const float *__restrict__ D = T.Ds32;
  float *G32 = T.Gacc32;
  float j12[NA * NB];
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) j12[x] = 0.f;
  const float dn_ab = T.screen ? __ldg(T.Dn32 + (size_t)bra.sa * nsh + bra.sb) : 0.f;
  const float *__restrict__ soa = T.soa32;
  const int np = T.npairs;
  const float *__restrict__ Dp = T.Dp32;          // pair-indexed ket data (null: n x n matrices)
  const float *__restrict__ DnP = T.DnP32;
  float *Jp = T.Jp32;
  const int kstride = T.nket;                     // element stride of the pair-indexed arrays
  unsigned cnt = 0;
  for (int k0 = warp * 32; k0 < nk; k0 += 32 * kRowWarps) {
    if (below_from(k0)) break;   // warp-uniform; every later ket chunk is below too
    const int kpos = k0 + lane;
    bool active = kpos < nk;
    const int kq = min(kpos, nk - 1);
    const int ki = T.ket0 + kq;
    PairRec32 ket;
    PrimRec32 kprim;
    if (soa) {
      // one coalesced 128-byte line per field and warp; only the fields the
      // class reads are loaded
      const float *f = soa + ki;
      ket.Q = f[kSoaQ * np];
      const int sh = __float_as_int(f[kSoaShells * np]), fn = __float_as_int(f[kSoaFuncs * np]);
      ket.sa = sh & 0xffff;
      ket.sb = sh >> 16;
      ket.fa = fn & 0xffff;
      ket.fb = fn >> 16;
      ket.nprim = 1;
      ket.prim0 = 0;
      if constexpr (LD > 0) {
        ket.AB[0] = f[kSoaABx * np];
        ket.AB[1] = f[kSoaABy * np];
        ket.AB[2] = f[kSoaABz * np];
      }
      kprim.p = f[kSoaP * np];
      kprim.Kt = f[kSoaKt * np];
      kprim.P[0] = f[kSoaPx * np];
      kprim.P[1] = f[kSoaPy * np];
      kprim.P[2] = f[kSoaPz * np];
      if constexpr (LC + LD > 0) {
        kprim.inv_p = f[kSoaInvP * np];
        kprim.PA[0] = f[kSoaPAx * np];
        kprim.PA[1] = f[kSoaPAy * np];
        kprim.PA[2] = f[kSoaPAz * np];
      }
    } else {
      ket = T.pairs32[ki];
    }
    float bound = bra.Q * ket.Q;
    if (T.screen) {
      float m = fmaxf(dn_ab, fmaxf(Dnab[ket.sa], Dnab[ket.sb]));
      m = fmaxf(m, DnP ? DnP[ki] : __ldg(T.Dn32 + (size_t)ket.sa * nsh + ket.sb));
      bound *= m;
      if (bound < cutoff) active = false;
    }
    if (!(bound < TL.split32)) active = false;   // the FP64 launch takes these
    const unsigned live = __ballot_sync(0xffffffffu, active);
    if (!live) continue;
    cnt += __popc(live);
    float I[Q::NINT];
    if (active) {
      if (soa)
        eri_quartet_k1<float, LA, LB, LC, LD>(bra, prims + bra.prim0, ket, kprim, TL.boys.f64, TL.boys.dd, I);
      else
        eri_quartet<float, LA, LB, LC, LD>(bra, prims + bra.prim0, ket, prims + ket.prim0, TL.boys.f64,
                                           TL.boys.dd, I);
    } else {
#pragma unroll
      for (int x = 0; x < Q::NINT; ++x) I[x] = 0.f;
    }
    const float deg = active ? pow2<float>((bra.sa != bra.sb) + (ket.sa != ket.sb) + (bi != ki)) : 0.f;
    const float hdeg = deg * hf;
    const int fc = ket.fa, fd = ket.fb;
    auto Iat = [&](int a, int b, int c, int d) -> float { return I[((a * NB + b) * NC + c) * ND + d]; };
    // J12 (bra block): D of the ket block, summed over this warp's kets
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        float dcd = 0.f;
        if (active) dcd = (Dp ? Dp[(size_t)(c * ND + d) * kstride + kq] : __ldg(D + (size_t)(fc + c) * n + fd + d)) * deg;
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int b = 0; b < NB; ++b) j12[a * NB + b] = fmaf(dcd, Iat(a, b, c, d), j12[a * NB + b]);
      }
    if (!active) continue;
    // the D rows of the bra shells at the ket's columns
    float dc[NC][NR], dd[ND][NR];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int r = 0; r < NR; ++r) dc[c][r] = Drow[(fc + c) * NRP + r];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
      for (int r = 0; r < NR; ++r) dd[d][r] = Drow[(fd + d) * NRP + r];
    // J34 (ket block): D of the bra block
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        float s = 0.f;
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int b = 0; b < NB; ++b) s = fmaf(Drow[(bra.fb + b) * NRP + a], Iat(a, b, c, d), s);
        if (Jp) atomicAdd(Jp + (size_t)(c * ND + d) * kstride + kq, s * deg);
        else atomicAdd(G32 + (size_t)(fc + c) * n + fd + d, s * deg);
      }
    // K13 (a,c) += D(b,d), K14 (a,d) += D(b,c): rows of shell a
#pragma unroll
    for (int a = 0; a < NA; ++a) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float s = 0.f;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
          for (int d = 0; d < ND; ++d) s = fmaf(dd[d][NA + b], Iat(a, b, c, d), s);
        atomicAdd(Krow + (fc + c) * NRP + a, s * hdeg);
      }
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        float s = 0.f;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
          for (int c = 0; c < NC; ++c) s = fmaf(dc[c][NA + b], Iat(a, b, c, d), s);
        atomicAdd(Krow + (fd + d) * NRP + a, s * hdeg);
      }
    }
    // K24 (b,d) += D(a,c), K23 (b,c) += D(a,d): rows of shell b
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        float s = 0.f;
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int c = 0; c < NC; ++c) s = fmaf(dc[c][a], Iat(a, b, c, d), s);
        atomicAdd(Krow + (fd + d) * NRP + NA + b, s * hdeg);
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        float s = 0.f;
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int d = 0; d < ND; ++d) s = fmaf(dd[d][a], Iat(a, b, c, d), s);
        atomicAdd(Krow + (fc + c) * NRP + NA + b, s * hdeg);
      }
    }
  }
  if (T.count && lane == 0 && cnt) atomicAdd(T.count, (unsigned long long)cnt);
  // J12: one reduction per warp
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) {
    const float v = warp_sum(j12[x]);
    if (lane == 0 && v != 0.f) atomicAdd(G32 + (size_t)(bra.fa + x / NB) * n + bra.fb + x % NB, v);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NRP * n; i += blockDim.x) {
    const float v = Krow[i];
    const int c = i / NRP, r = i - c * NRP;
    if (v != 0.f && r < NR) atomicAdd(G32 + (size_t)(r < NA ? bra.fa + r : bra.fb + (r - NA)) * n + c, v);
  }
}

// ---------------------------------------------------------------- coupling --
// Bra pairs of species A (every unordered shell pair), ket pairs of species B.
// J_A[i][j] += scale sum_{kl} D_B[k][l] (ij|kl), J_B[k][l] += scale
// sum_{ij} D_A[i][j] (ij|kl), both as full symmetric matrices; raw |v| < cut is
// dropped (the reference's 1e-10 test on each integral).
// A warp keeps its bra pair and walks up to TL.tile.chunk ket tiles; J_A is
// summed over them before its one reduction.
// No double-float tier: the launches are short, and two per class took 306 us
// where one takes 249 (six waters).
template <typename R, int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) cp_tasks_kernel(const CPTask *__restrict__ tasks, TaskLaunch TL) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr bool F64 = std::is_same<R, double>::value;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  const int t = find_task(tasks, TL.ntasks, blockIdx.x);
  const CPTask &T = tasks[t];
  const int act = system_flag(T.active);
  if (act == kSysOff) return;   // converged system: nothing to build
  if (act == kSysFP64 && TL.mixed && TL.lower) return;   // system held in FP64: the FP64 launch takes it all
  const int local = blockIdx.x - T.blk0;
  const int kets = TL.tile.kets, parts = 32 / kets;
  const int ty = local / T.nbx;
  const int kl = threadIdx.x & (kets - 1), part = parts == 1 ? 0 : threadIdx.x / kets;
  const int bpos = ty * blockDim.y + threadIdx.y;
  if (bpos >= T.nbra) return;
  const int bi = T.bra0 + bpos;
  int k0 = (local - ty * T.nbx) * TL.tile.chunk * kets;
  const int kend = min(T.nket, k0 + TL.tile.chunk * kets);
  const float qbra = T.pa32[bi].Q;
  // |(ij|kl)| <= Q_ab Q_cd for every component (Schwarz), and raw values below
  // the cut are dropped, so a quartet below it contributes nothing.  Pairs are
  // sorted by decreasing Schwarz factor: the first ket of a tile bounds all
  // after it (0.99999: room for the FP32 rounding of the factors).
  const float reach = 0.99999f * TL.cut32;
  if (qbra * T.pb32[T.ket0 + k0].Q < reach) return;
  const PairT<R> *pa, *pb;
  const PrimT<R> *pra, *prb;
  if constexpr (F64) {
    pa = T.pa; pb = T.pb; pra = T.pra; prb = T.prb;
  } else {
    pa = T.pa32; pb = T.pb32; pra = T.pra32; prb = T.prb32;
  }
  auto DA = [&](int i) { return elem<R>(T.DsA, T.DsA32, nullptr, i); };
  auto DB = [&](int i) { return elem<R>(T.DsB, T.DsB32, nullptr, i); };
  R scale, cut;
  if constexpr (F64) {
    scale = T.scale;
    cut = TL.cut;
  } else {
    scale = T.scale32;
    cut = TL.cut32;
  }
  const PairT<R> &bra = pa[bi];
  const int fa = bra.fa, fb = bra.fb, nA = T.nA, nB = T.nB;
  const bool abdiff = bra.sa != bra.sb;
  R ja[NA * NB];
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) ja[x] = R(0);
  unsigned cnt = 0;
  for (; k0 < kend; k0 += kets) {
    if (qbra * T.pb32[T.ket0 + k0].Q < reach) break;
    const int kpos = k0 + kl;
    bool active = kpos < T.nket;
    const int ki = T.ket0 + min(kpos, T.nket - 1);
    const PairRec32 &k32 = T.pb32[ki];
    const float qq = qbra * k32.Q;
    if (TL.mixed) {
      // the test is done in FP32 in mixed launches so both launches agree; FP32
      // for quartets whose Q_ab Q_cd max(|D_A|, |D_B|) bound (FP32, identical in
      // both launches) is below the split
      if (qq * 0.999f < TL.cut32) active = false;
      const PairRec32 &b32 = T.pa32[bi];
      float dm = 0.f;
      if (T.DnA32) dm = __ldg(T.DnA32 + b32.sa * T.nshA + b32.sb);
      if (T.DnB32) dm = fmaxf(dm, __ldg(T.DnB32 + k32.sa * T.nshB + k32.sb));
      const float b = qq * dm;
      if (act != kSysFP64 && (TL.lower ? !(b < TL.split32) : (b < TL.split32))) active = false;
      if ((T.DnA32 || T.DnB32) && act != kSysFP64 && b < TL.skip) active = false;
    } else if (qq < 1.00001f * TL.cut32) {
      // too near the cut for FP32 to decide
      if (qq < 0.99999f * TL.cut32 || abs_below(T.pa[bi].Q * T.pb[ki].Q * (1.0 - 1e-9), TL.cut)) active = false;
    }
    if (!__any_sync(0xffffffffu, active)) continue;
    cnt += __popc(__ballot_sync(0xffffffffu, active && part == 0));
    const PairT<R> &ket = pb[ki];
    R I[Q::NINT];
    if (active || parts > 1) {
      eri_quartet<R, LA, LB, LC, LD>(bra, pra + bra.prim0, ket, prb + ket.prim0, TL.boys.f64, TL.boys.dd, I, part, parts,
                                     active);
      if (part) active = false;   // the quartet is digested by its first lane
    }
    if (active) {
#pragma unroll
      for (int x = 0; x < Q::NINT; ++x)
        if (abs_below(I[x], cut)) I[x] = R(0);
      const int fc = ket.fa, fd = ket.fb;
      const bool cddiff = ket.sa != ket.sb;
      if (T.JA) {
        const R wk = cddiff ? scale + scale : scale;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            const R w = wk * DB((fc + c) * nB + fd + d);
#pragma unroll
            for (int x = 0; x < NA * NB; ++x) ja[x] = mad(w, I[(x * NC + c) * ND + d], ja[x]);
          }
      }
      if (T.JB) {
        const R wb = abdiff ? scale + scale : scale;
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int d = 0; d < ND; ++d) {
            R s = R(0);
#pragma unroll
            for (int x = 0; x < NA * NB; ++x)
              s = mad(DA((fa + x / NB) * nA + fb + x % NB), I[(x * NC + c) * ND + d], s);
            s = s * wb;
            atomic_acc<R>(T.JB, T.JB32, (size_t)(fc + c) * nB + fd + d, s);
            if (cddiff) atomic_acc<R>(T.JB, T.JB32, (size_t)(fd + d) * nB + fc + c, s);
          }
      }
    }
    __syncwarp();
  }
  if (!cnt) return;   // warp-uniform
  if (T.JA)
#pragma unroll
    for (int x = 0; x < NA * NB; ++x) {
      const R s = warp_sum(ja[x]);
      if (threadIdx.x == 0) {
        atomic_acc<R>(T.JA, T.JA32, (size_t)(fa + x / NB) * nA + fb + x % NB, s);
        if (abdiff) atomic_acc<R>(T.JA, T.JA32, (size_t)(fb + x % NB) * nA + fa + x / NB, s);
      }
    }
  if (T.count && threadIdx.x == 0) atomicAdd(T.count, (unsigned long long)cnt);
}

// ----------------------------------------------------------- geminal (G12) --
// Matrices of a geminal pair potential, one quartet per lane over the launch's
// bra x ket pairs (no screening): the six updates of one species, or J of the
// bra species with raw |v| < cut dropped.  FP64 bound (an exponential and a
// reciprocal square root per term and primitive quartet); two waters (68
// functions, three terms): 3.10 ms with one quartet per warp on the cooperative
// kernel, 0.20 ms so.
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) g12_kernel(G12Params P) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  const int kets = P.kets, parts = 32 / kets, part = threadIdx.x / kets, bras = blockDim.y;
  if (P.triangle && blockIdx.x * kets > blockIdx.y * bras + bras - 1) return;
  const int kpos = blockIdx.x * kets + (threadIdx.x & (kets - 1));
  const int bpos = blockIdx.y * bras + threadIdx.y;
  if (bpos >= P.nbra) return;   // warp-uniform
  bool active = kpos < P.nket && !(P.triangle && kpos > bpos);
  if (!__any_sync(0xffffffffu, active)) return;
  const int bi = P.bra0 + bpos, ki = P.ket0 + min(kpos, P.nket - 1);
  const PairRec &bra = P.pa[bi];
  const PairRec &ket = P.pb[ki];
  double I[Q::NINT];
  eri_quartet<double, LA, LB, LC, LD, true>(bra, P.pra + bra.prim0, ket, P.prb + ket.prim0, P.gem, nullptr, I, part,
                                            parts, active);
  if (part) active = false;   // the quartet is digested by its first lane
  const int fa = bra.fa, fb = bra.fb, fc = ket.fa, fd = ket.fb, n = P.n;
  double j12[NA * NB];
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) j12[x] = 0.0;
  if (active) {
    if (P.intra) {
      const double deg = pow2<double>((bra.sa != bra.sb) + (ket.sa != ket.sb) + (bi != ki));
      jk_digest<double, LA, LB, LC, LD>(I, [&](int i) { return __ldg(P.Ds + i); }, n, fa, fb, fc, fd, deg, P.hf * deg,
                                        P.Gacc, nullptr, j12);
    } else {
      const double two = ket.sa != ket.sb ? 2.0 : 1.0;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const double w = two * __ldg(P.Ds + (size_t)(fc + c) * P.nB + fd + d);
#pragma unroll
          for (int x = 0; x < NA * NB; ++x) {
            const double v = I[(x * NC + c) * ND + d];
            if (!abs_below(v, P.cut)) j12[x] = fma(w, v, j12[x]);
          }
        }
    }
  }
  __syncwarp();
  const bool both = !P.intra && bra.sa != bra.sb;
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) {
    const double v = warp_sum(j12[x]);
    if (threadIdx.x == 0) {
      atomicAdd(P.Gacc + (size_t)(fa + x / NB) * n + fb + x % NB, v);
      if (both) atomicAdd(P.Gacc + (size_t)(fb + x % NB) * n + fa + x / NB, v);
    }
  }
}

// ------------------------------------------------------- first quarter (IT) --
// Output A[nu][lam][sig] accumulates sum_mu Cs(mu) v(mu nu|lam sig) over every
// distinct member of the quartet's permutational orbit (intra) or of the
// (bra swap) x (ket swap) orbit (coupling); v are raw integrals with |v| > cut.
template <int NMU, int NNU, int NL, int NS, typename F>
__device__ __forceinline__ void it_role(F &&val, const double *__restrict__ Cs, int fmu, int fnu, int fl, int fs,
                                        double *A, int nB) {
#pragma unroll
  for (int nu = 0; nu < NNU; ++nu)
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        double acc = 0;
#pragma unroll
        for (int mu = 0; mu < NMU; ++mu) acc += __ldg(Cs + fmu + mu) * val(mu, nu, l, s);
        atomicAdd(A + ((size_t)(fnu + nu) * nB + fl + l) * nB + fs + s, acc);
      }
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) it_kernel(ITParams P) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  const int kets = P.kets, parts = 32 / kets, bras = blockDim.y;
  if (P.triangle && blockIdx.x * kets > blockIdx.y * bras + bras - 1) return;
  const int part = threadIdx.x / kets;
  const int kpos = blockIdx.x * kets + (threadIdx.x & (kets - 1));
  const int bpos = blockIdx.y * bras + threadIdx.y;
  if (bpos >= P.nbra) return;   // warp-uniform
  const int bi = P.bra0 + bpos, ki = P.ket0 + min(kpos, P.nket - 1);
  const PairRec bra = P.pa[bi];
  const PairRec ket = P.pb[ki];
  // every raw integral is bounded by Q_ab Q_cd (Schwarz) and only |v| > cut is used
  bool active = kpos < P.nket && !(P.triangle && kpos > bpos) && abs_above(bra.Q * ket.Q * (1.0 - 1e-9), P.cut);
  if (P.screen && active) {
    const double b = bra.Q * ket.Q * dnorm6(P.Dn, P.nsh, bra.sa, bra.sb, ket.sa, ket.sb);
    if (abs_below(b, P.eps)) active = false;
  }
  if (parts == 1 ? !active : __all_sync(0xffffffffu, !active)) return;
  double I[Q::NINT];
  eri_quartet<double, LA, LB, LC, LD>(bra, P.pra + bra.prim0, ket, P.prb + ket.prim0, P.boys.f64, P.boys.dd, I, part,
                                      parts, active);
  if (part || !active) return;
#pragma unroll
  for (int x = 0; x < Q::NINT; ++x)
    if (!abs_above(I[x], P.cut)) I[x] = 0.0;
  auto I4 = [&](int a, int b, int c, int d) -> double { return I[((a * NB + b) * NC + c) * ND + d]; };
  const bool ab = bra.sa != bra.sb, cd = ket.sa != ket.sb;
  const int fa = bra.fa, fb = bra.fb, fc = ket.fa, fd = ket.fb, nB = P.nB;
  const double *Cs = P.Cs;
  // (a b|c d): mu=a nu=b
  it_role<NA, NB, NC, ND>([&](int mu, int nu, int l, int s) { return I4(mu, nu, l, s); }, Cs, fa, fb, fc, fd, P.A, nB);
  if (ab)
    it_role<NB, NA, NC, ND>([&](int mu, int nu, int l, int s) { return I4(nu, mu, l, s); }, Cs, fb, fa, fc, fd, P.A, nB);
  if (cd)
    it_role<NA, NB, ND, NC>([&](int mu, int nu, int l, int s) { return I4(mu, nu, s, l); }, Cs, fa, fb, fd, fc, P.A, nB);
  if (ab && cd)
    it_role<NB, NA, ND, NC>([&](int mu, int nu, int l, int s) { return I4(nu, mu, s, l); }, Cs, fb, fa, fd, fc, P.A, nB);
  if (P.intra && bi != ki) {
    // (c d|a b) and its swaps: mu in the ket pair
    it_role<NC, ND, NA, NB>([&](int mu, int nu, int l, int s) { return I4(l, s, mu, nu); }, Cs, fc, fd, fa, fb, P.A, nB);
    if (cd)
      it_role<ND, NC, NA, NB>([&](int mu, int nu, int l, int s) { return I4(l, s, nu, mu); }, Cs, fd, fc, fa, fb, P.A, nB);
    if (ab)
      it_role<NC, ND, NB, NA>([&](int mu, int nu, int l, int s) { return I4(s, l, mu, nu); }, Cs, fc, fd, fb, fa, P.A, nB);
    if (ab && cd)
      it_role<ND, NC, NB, NA>([&](int mu, int nu, int l, int s) { return I4(s, l, nu, mu); }, Cs, fd, fc, fb, fa, P.A, nB);
  }
}

// ------------------------------------------------------ MP2 transform input --
// Warp y: (lam sig) pair tile_y * bras + y of the batch; its lanes: (mu nu) pairs
// tile_x * kets + (lane mod kets), 32 / kets lanes each.
// R = dd32 writes the split-BF16 form only, whose pieces hold an integral to 2^-16 or
// 2^-24 of itself.  A double-float integral is within 2^-41 Q_ab Q_cd of the FP64 one,
// 2^-43 in the middle: at least 2^17 below the rounding of the quartet's largest
// integral to 24 bits, and so below what that does to any (ia|jb).  An integral
// that its terms cancel down to the cut may have fewer than 24 correct bits
// there, and weighs as little: E_MP2 of twelve waters with d is the same to the
// last digit with FP64 integrals (116.3 ms; double-float 114.4; four waters in a
// contracted basis 7.4 and 5.0 ms).
template <typename R, int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128, jk_min_blocks<R, LA, LB, LC, LD>()) mp2x_kernel(MXParams P) {
  if (beside_block()) return;
  using Q = QClass<LA, LB, LC, LD>;
  constexpr bool DD = std::is_same<R, dd32>::value;
  constexpr int NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  const int kets = P.kets, parts = 32 / kets, part = parts == 1 ? 0 : threadIdx.x / kets;
  const int kpos = blockIdx.x * kets + (threadIdx.x & (kets - 1));
  const int bpos = blockIdx.y * blockDim.y + threadIdx.y;
  if (bpos >= P.nbra) return;   // warp-uniform
  const int bi = P.bra0 + bpos, ki = P.ket0 + min(kpos, P.nket - 1);
  bool active = kpos < P.nket;
  // quartet selection as in FP64; where the FP32 factors decide beyond their
  // rounding (Q and norms: 4e-7), without an FP64 instruction
  auto keeps = [&]() {
    const double qq = P.pairs[bi].Q * P.kpairs[ki].Q;
    if (!abs_above(qq * (1.0 - 1e-9), P.cut)) return false;
    const PairRec &x = P.pairs[bi], &y = P.kpairs[ki];
    return !(P.screen && abs_below(qq * dnorm6(P.Dn, P.nsh, x.sa, x.sb, y.sa, y.sb), P.eps));
  };
  const PairT<R> *pb, *pk;
  const PrimT<R> *rb, *rk;
  if constexpr (DD) {
    pb = P.pairsd; pk = P.kpairsd; rb = P.primsd; rk = P.kprimsd;
    const float qq = pb[bi].Q.hi * pk[ki].Q.hi, cut = (float)P.cut;
    if (qq < 0.99999f * cut) active = false;
    else if (active && (P.screen || qq < 1.00001f * cut)) active = keeps();
  } else {
    pb = P.pairs; pk = P.kpairs; rb = P.prims; rk = P.kprims;
    if (active) active = keeps();
  }
  if (parts == 1 ? !active : __all_sync(0xffffffffu, !active)) return;
  const PairT<R> &bra = pb[bi];
  const PairT<R> ket = pk[ki];
  R I[Q::NINT];
  eri_quartet<R, LA, LB, LC, LD>(bra, rb + bra.prim0, ket, rk + ket.prim0, P.boys.f64, P.boys.dd, I, part, parts, active);
  if (part || !active) return;
  const int col0 = __ldg(P.colbase + bi) - P.col_first;
  const bool two = ket.sa != ket.sb;
  const size_t n = P.n, ncol = P.ncol;
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          const R v = I[((a * NB + b) * NC + c) * ND + d];
          if (!above_cut(v, P.cut)) continue;
          const size_t col = col0 + a * NB + b;
          if constexpr (!DD) {
            if (P.X) {
              P.X[((ket.fa + c) * ncol + col) * n + ket.fb + d] = v;
              if (two) P.X[((ket.fb + d) * ncol + col) * n + ket.fa + c] = v;
              continue;
            }
          }
          // Xt[col * Kp + nu][mu] and the mirrored bra orientation
          float x;
          if constexpr (DD) x = fadd(v.hi, v.lo);
          else x = (float)v;
          __nv_bfloat16 pc[kMaxPieces];
          bf16_pieces(x, P.np, pc);   // three pieces hold the FP32 value exactly
          const size_t kp = P.Kp;
          const size_t j1 = (col * kp + ket.fb + d) * kp + ket.fa + c;
          const size_t j2 = (col * kp + ket.fa + c) * kp + ket.fb + d;
          for (int k = 0; k < P.np; ++k) {
            P.Xp[k][j1] = pc[k];
            if (two) P.Xp[k][j2] = pc[k];
          }
        }
}

}  // namespace lgb
