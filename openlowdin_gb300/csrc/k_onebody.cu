// One-electron matrices on the device: overlap S, kinetic T and the
// point-charge potential V = sum_C Z_C <a|1/|r - C||b> of one species,
// Obara-Saika recursions (1-D overlap tables for S and T; the vertical recursion
// with Boys values and a horizontal transfer for V), written normalised
// (norma_i norma_j) to both (i, j) and (j, i).  S and T: one thread per unordered
// shell pair.  V of s, p and d shells: potential_kernel, a group of lanes per
// pair with the charges dealt to them and every index a compile-time constant.
// V is FP64 bound and grows with the charges: for a 387-function chain and its
// nuclei one thread per pair with run-time indices took 326 us in 244 blocks,
// all launches together now take 226.  Same formulas as the host blocks the
// library's LibintInterface_compute_1body_ints uses (ContractedGaussian /
// Overlap / Kinetic / Attraction integrals of the reference, src/ints/*.f90).
#include "eri.cuh"
#include "eri_generic.cuh"
#include "kernels.cuh"

namespace lgb {
namespace {

constexpr int kOneMaxL = kMaxL + 2;   // kinetic needs j + 2
constexpr int kPotMaxL = 2;           // shells of potential_kernel

// V of the pairs whose later shell has angular momentum LA and whose earlier one
// (or the same) LB: `lanes` (a power of two) neighbouring lanes
// per pair, lane g evaluating charges g, g + lanes, ...; shells of angular
// momentum l are P.order[P.lstart[l]] .. P.order[P.lstart[l + 1] - 1].  The
// charges' terms pass through shared memory and are added in the order of the
// charges, one element of the pair per lane, so the result does not depend on
// the number of lanes: the sums are those of one thread taking one charge after
// the other, to the bit.
template <int LA, int LB>
__global__ void __launch_bounds__(128) potential_kernel(OneBodyParams P, int lanes) {
  if (beside_block()) return;
  constexpr int L = LA + LB, NE = coff(L + 1), E0 = coff(LA), nE = NE - E0, NA = ncart(LA), NB = ncart(LB);
  __shared__ double term[128][nE + 1];   // per lane: W of its charge, then Z w
  __shared__ double sum[128][nE];        // per group (at its first lane): contracted X
  const int na = P.lstart[LA + 1] - P.lstart[LA], nb = P.lstart[LB + 1] - P.lstart[LB];
  const int npair = LA == LB ? na * (na + 1) / 2 : na * nb;
  const int t = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / lanes), g = threadIdx.x & (lanes - 1);
  if (t >= npair) return;   // a whole group
  const int base = threadIdx.x - g;
  const unsigned group = (lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1u)) << (base & 31);
  int ia, ib;
  if constexpr (LA == LB) {
    ia = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while (ia * (ia + 1) / 2 > t) --ia;
    while ((ia + 1) * (ia + 2) / 2 <= t) ++ia;
    ib = t - ia * (ia + 1) / 2;
  } else {
    ia = t / nb;
    ib = t - ia * nb;
  }
  const int oa = P.order[P.lstart[LA] + ia], ob = P.order[P.lstart[LB] + ib];
  if (oa < ob) return;   // the pair belongs to the class (LB LA)
  const DevShell A = P.shells[oa], B = P.shells[ob];
  double AB[3], AB2 = 0;
  for (int d = 0; d < 3; ++d) {
    AB[d] = A.O[d] - B.O[d];
    AB2 += AB[d] * AB[d];
  }
  for (int e = g; e < nE; e += lanes) sum[base][e] = 0.0;
  for (int pa = 0; pa < A.nprim; ++pa)
    for (int pb = 0; pb < B.nprim; ++pb) {
      const double a = P.alpha[A.p0 + pa], b = P.alpha[B.p0 + pb], p = a + b, o2p = 0.5 / p;
      const double cab = P.cn[A.p0 + pa] * P.cn[B.p0 + pb] * exp(-a * b / p * AB2);
      double Pc[3], PA[3];
      for (int d = 0; d < 3; ++d) {
        Pc[d] = (a * A.O[d] + b * B.O[d]) / p;
        PA[d] = Pc[d] - A.O[d];
      }
      const double w = cab * 2.0 * 3.14159265358979323846 / p;
      for (int c0 = 0; c0 < P.ncharge; c0 += lanes) {
        const int c = c0 + g;
        if (c < P.ncharge) {
          double PC[3], PC2 = 0, F[L + 1];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            PC[d] = Pc[d] - P.R[3 * c + d];
            PC2 += PC[d] * PC[d];
          }
          boys_f64_rt(L, p * PC2, F, P.boys.f64);
          double W[NE][L + 1];
#pragma unroll
          for (int m = 0; m <= L; ++m) W[0][m] = F[m];
          sfor<1, NE>([&](auto ec) {
            constexpr int e = decltype(ec)::value;
            constexpr int d = cdir(e), em = cminus(e, d), ei = ccomp(e, d) - 1;
            constexpr int emm = ei > 0 ? cminus(em, d) : 0;
#pragma unroll
            for (int m = 0; m <= L - clevel(e); ++m) {
              double v = PA[d] * W[em][m] - PC[d] * W[em][m + 1];
              if constexpr (ei > 0) v += ei * o2p * (W[emm][m] - W[emm][m + 1]);
              W[e][m] = v;
            }
          });
          sfor<E0, NE>([&](auto ec) {
            constexpr int e = decltype(ec)::value;
            term[threadIdx.x][e - E0] = W[e][0];
          });
          term[threadIdx.x][nE] = P.Z[c] * w;
        }
        __syncwarp(group);
        const int cnt = min(lanes, P.ncharge - c0);
        for (int e = g; e < nE; e += lanes) {
          double x = sum[base][e];
          for (int j = 0; j < cnt; ++j) x += term[base + j][nE] * term[base + j][e];
          sum[base][e] = x;
        }
        __syncwarp(group);
      }
    }
  if (g) return;
  double X[nE], V[NA * NB];
#pragma unroll
  for (int e = 0; e < nE; ++e) X[e] = sum[base][e];
  hrr<double, LA, LB, 1>(X, AB, V);
  const int fa = P.first[oa], fb = P.first[ob];
  const size_t n = P.n;
#pragma unroll
  for (int x = 0; x < NA * NB; ++x) {
    const int i = fa + x / NB, j = fb + x % NB;
    const double nn = P.norma[i] * P.norma[j];
    P.V[i * n + j] = P.V[j * n + i] = V[x] * nn;
  }
}

__device__ void ovl1d_dev(int li, int lj, double PA, double PB, double o2p, double s[kMaxL + 1][kOneMaxL + 1]) {
  for (int i = 0; i <= li; ++i)
    for (int j = 0; j <= lj; ++j) {
      double v;
      if (!i && !j) {
        v = 1.0;
      } else if (i > 0) {
        v = PA * s[i - 1][j];
        if (i > 1) v += (i - 1) * o2p * s[i - 2][j];
        if (j > 0) v += j * o2p * s[i - 1][j - 1];
      } else {
        v = PB * s[0][j - 1];
        if (j > 1) v += (j - 1) * o2p * s[0][j - 2];
      }
      s[i][j] = v;
    }
}

// S and T of every pair, or (WITHV) V of the pairs with an f shell: apart, so that
// the chains of the two run beside one another (three waters with an f shell on
// O: 1.04 ms in one kernel, 0.81 so; one thread per pair for everything took 0.94)
template <bool WITHV>
__global__ void __launch_bounds__(128) one_body_kernel(OneBodyParams P) {
  if (beside_block()) return;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int npair = P.nsh * (P.nsh + 1) / 2;
  if (t >= npair) return;
  // t -> (s1 >= s2)
  int s1 = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
  while (s1 * (s1 + 1) / 2 > t) --s1;
  while ((s1 + 1) * (s1 + 2) / 2 <= t) ++s1;
  const int s2 = t - s1 * (s1 + 1) / 2;
  const DevShell A = P.shells[s1], B = P.shells[s2];
  const CartInfo *ct = kCartTable.e;
  const int la = A.l, lb = B.l, n1 = ncart(la), n2 = ncart(lb);
  const bool dov = WITHV && (la > kPotMaxL || lb > kPotMaxL);
  constexpr int kNC2 = ncart(kMaxL) * ncart(kMaxL);
  double S[kNC2], T[kNC2], V[kNC2];
  for (int k = 0; k < n1 * n2; ++k) S[k] = T[k] = V[k] = 0.0;
  double AB[3], AB2 = 0;
  for (int d = 0; d < 3; ++d) {
    AB[d] = A.O[d] - B.O[d];
    AB2 += AB[d] * AB[d];
  }
  // potential: vertical recursion on the bra up to la + lb, then transfer
  const int L = la + lb, NE = coff(L + 1), E0 = coff(la), M = L + 1;
  double W[coff(2 * kMaxL + 1) * (2 * kMaxL + 1)], X[coff(2 * kMaxL + 1)];
  if (dov)
    for (int e = 0; e < NE - E0; ++e) X[e] = 0.0;
  for (int pa = 0; pa < A.nprim; ++pa)
    for (int pb = 0; pb < B.nprim; ++pb) {
      const double a = P.alpha[A.p0 + pa], b = P.alpha[B.p0 + pb], p = a + b, o2p = 0.5 / p;
      const double cab = P.cn[A.p0 + pa] * P.cn[B.p0 + pb] * exp(-a * b / p * AB2);
      double Pc[3], PA[3];
      for (int d = 0; d < 3; ++d) {
        Pc[d] = (a * A.O[d] + b * B.O[d]) / p;
        PA[d] = Pc[d] - A.O[d];
      }
      if (P.S || P.T) {
        const double pref = cab * pow(3.14159265358979323846 / p, 1.5);
        double s[3][kMaxL + 1][kOneMaxL + 1];
        for (int d = 0; d < 3; ++d) ovl1d_dev(la, lb + 2, PA[d], Pc[d] - B.O[d], o2p, s[d]);
        for (int f1 = 0; f1 < n1; ++f1) {
          const CartInfo &c1 = ct[coff(la) + f1];
          for (int f2 = 0; f2 < n2; ++f2) {
            const CartInfo &c2 = ct[coff(lb) + f2];
            const double sx = s[0][c1.xyz[0]][c2.xyz[0]], sy = s[1][c1.xyz[1]][c2.xyz[1]],
                         sz = s[2][c1.xyz[2]][c2.xyz[2]];
            S[f1 * n2 + f2] += pref * sx * sy * sz;
            double tk[3];
            for (int d = 0; d < 3; ++d) {
              const int i = c1.xyz[d], j = c2.xyz[d];
              double v = -2.0 * b * (2 * j + 1) * s[d][i][j] + 4.0 * b * b * s[d][i][j + 2];
              if (j >= 2) v += j * (j - 1) * s[d][i][j - 2];
              tk[d] = -0.5 * v;
            }
            T[f1 * n2 + f2] += pref * (tk[0] * sy * sz + sx * tk[1] * sz + sx * sy * tk[2]);
          }
        }
      }
      if (dov) {
        const double w = cab * 2.0 * 3.14159265358979323846 / p;
        for (int c = 0; c < P.ncharge; ++c) {
          double PC[3], PC2 = 0, F[kGenMaxL + 1];
          for (int d = 0; d < 3; ++d) {
            PC[d] = Pc[d] - P.R[3 * c + d];
            PC2 += PC[d] * PC[d];
          }
          boys_f64_rt(L, p * PC2, F, P.boys.f64);
          for (int m = 0; m <= L; ++m) W[m] = F[m];
          for (int e = 1; e < NE; ++e) {
            const CartInfo &ce = ct[e];
            const int d = ce.dir, em = ce.m[d], ei = ce.xyz[d] - 1;
            for (int m = 0; m <= L - ce.lev; ++m) {
              double v = PA[d] * W[em * M + m] - PC[d] * W[em * M + m + 1];
              if (ei > 0) {
                const int emm = ct[em].m[d];
                v += ei * o2p * (W[emm * M + m] - W[emm * M + m + 1]);
              }
              W[e * M + m] = v;
            }
          }
          const double zw = P.Z[c] * w;
          for (int e = E0; e < NE; ++e) X[e - E0] += zw * W[e * M];
        }
      }
    }
  if (dov) {
    // horizontal transfer (a, b+1_i| = (a+1_i, b| + AB_i (a, b| over lb
    // levels: level j has rows over totals la .. la + lb - j (the last level
    // only la) and ncart(j) columns; it reads level j - 1 (X for j = 1)
    constexpr int kHRows = coff(2 * kMaxL), kHCols = ncart(kMaxL);
    double Hb[2][kHRows * kHCols];
    if (lb == 0) {
      for (int f1 = 0; f1 < n1; ++f1) V[f1] = X[f1];
    } else {
      for (int j = 1; j <= lb; ++j) {
        const int na = j == lb ? n1 : coff(la + lb - j + 1) - E0, nb = ncart(j), pnb = j == 1 ? 1 : ncart(j - 1);
        const double *src = j == 1 ? X : Hb[j & 1];
        double *dst = j == lb ? V : Hb[(j - 1) & 1];
        for (int bi = 0; bi < nb; ++bi) {
          const int bc = coff(j) + bi, d = ct[bc].dir, bm = ct[bc].m[d] - coff(j - 1);
          for (int ar = 0; ar < na; ++ar) {
            const int apr = ct[E0 + ar].p[d] - E0;
            dst[ar * nb + bi] = src[apr * pnb + bm] + AB[d] * src[ar * pnb + bm];
          }
        }
      }
    }
  }
  const int fa = P.first[s1], fb = P.first[s2];
  const size_t n = P.n;
  for (int f1 = 0; f1 < n1; ++f1)
    for (int f2 = 0; f2 < n2; ++f2) {
      const int i = fa + f1, j = fb + f2;
      const double nn = P.norma[i] * P.norma[j];
      const int k = f1 * n2 + f2;
      if (P.S) P.S[i * n + j] = P.S[j * n + i] = S[k] * nn;
      if (P.T) P.T[i * n + j] = P.T[j * n + i] = T[k] * nn;
      if (dov) P.V[i * n + j] = P.V[j * n + i] = V[k] * nn;
    }
}

}  // namespace

cudaError_t launch_one_body(const OneBodyParams &p, Queue &q) {
  const int npair = p.nsh * (p.nsh + 1) / 2;
  if (npair <= 0 || (!p.S && !p.T)) return cudaSuccess;
  count_launches(q.sizing ? 0 : 1);
  return launch_beside(q, &one_body_kernel<false>, (npair + 127) / 128, 128, 0, p);
}

cudaError_t launch_potential_f(OneBodyParams p, Queue &q) {
  const int npair = p.nsh * (p.nsh + 1) / 2;
  if (npair <= 0 || !p.V || p.ncharge <= 0 || p.lstart[kPotMaxL + 1] >= p.nsh) return cudaSuccess;
  count_launches(q.sizing ? 0 : 1);
  p.S = p.T = nullptr;
  return launch_beside(q, &one_body_kernel<true>, (npair + 127) / 128, 128, 0, p);
}

cudaError_t launch_potential(int la, int lb, const OneBodyParams &p, Queue &q) {
  using Fn = void (*)(OneBodyParams, int);
  static const Fn fn[3][3] = {{&potential_kernel<0, 0>, &potential_kernel<0, 1>, &potential_kernel<0, 2>},
                              {&potential_kernel<1, 0>, &potential_kernel<1, 1>, &potential_kernel<1, 2>},
                              {&potential_kernel<2, 0>, &potential_kernel<2, 1>, &potential_kernel<2, 2>}};
  static_assert(kPotMaxL == 2, "one entry per class of potential_kernel");
  const long long npair = potential_pairs(la, lb, p);
  if (npair <= 0 || p.ncharge <= 0) return cudaSuccess;
  // lanes per pair: up to four warps per scheduler, no more than there are charges
  int lanes = 1;
  while (lanes < 32 && 2 * lanes <= p.ncharge && npair / 32 * lanes < 2 * (long long)kFillWarps) lanes *= 2;
  count_launches(q.sizing ? 0 : 1);
  return launch_beside(q, fn[la][lb], (unsigned)((npair * lanes + 127) / 128), 128, 0, p, lanes);
}

long long potential_pairs(int la, int lb, const OneBodyParams &p) {
  if (la < 0 || lb < 0 || la > kPotMaxL || lb > kPotMaxL) return 0;
  const long long na = p.lstart[la + 1] - p.lstart[la], nb = p.lstart[lb + 1] - p.lstart[lb];
  return la == lb ? na * (na + 1) / 2 : na * nb;
}

}  // namespace lgb
