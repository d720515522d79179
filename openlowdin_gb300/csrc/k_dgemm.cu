// FP64 matrix products of the MP2 transform on the FP64 tensor instruction
// (mma.m8n8k4, the only FP64 matrix instruction of this part; tcgen05 has none).
//
//   C_z[m][n] = sum_k A_z[m][k] B_z[k][n], any strides, z < batch.
//
// The instruction runs on the FP64 pipe, which these kernels keep 95 % busy (1.1
// TFLOP/s on dense operands), so operands
// straight from global memory and L1 keep up with it and nothing is staged.
// What matters is to issue no padded products and to keep every scheduler
// supplied: the occupied-index products have M = 16 to 64 rows against 10^4 to
// 10^6 columns, for which a library tile of 32 or 64 rows spent half its work
// on padding.  A warp owns a tile of 8 MB rows and 8 NB columns; MB is the row
// count in eighths, divided evenly over the row chunks.  Four waters with d (n
// 160, 16 occupied, 140 virtual, 13,696 columns), library -> here: first
// quarter 10.2 -> 5.1 ms, second 5.2 -> 4.6, third and fourth 0.56 -> 0.23 ms
// per occupied orbital.  The whole of E_MP2 against the library's products: 8 to
// 16 waters with d (320 to 640 functions) 411 -> 399, 1162 -> 933, 2497 -> 2138 and
// 7705 -> 7648 ms.
#include "kernels.cuh"

namespace lgb {
namespace {

struct DGemmArgs {
  int M, N, K;
  const double *A, *B;
  double *C;
  long long sam, sak, sbk, sbn, scm, scn;   // element strides
  long long za, zb, zc;                     // batch strides
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// lane l: A element (row l / 4, k l % 4), B element (k l % 4, column l / 4),
// C elements (row l / 4, columns 2 (l % 4) and the next)
template <int MB, int NB>
__global__ void __launch_bounds__(128) dgemm_kernel(DGemmArgs g) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const long long tile = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long n0 = tile * (8 * NB);
  if (n0 >= g.N) return;   // a whole warp
  const int m0 = blockIdx.y * (8 * MB);
  const double *A = g.A + blockIdx.z * g.za, *B = g.B + blockIdx.z * g.zb;
  // rows and columns beyond the matrix read its last one; they are not stored
  const double *pa[MB], *pb[NB];
#pragma unroll
  for (int i = 0; i < MB; ++i) pa[i] = A + (long long)min(m0 + 8 * i + r, g.M - 1) * g.sam;
#pragma unroll
  for (int j = 0; j < NB; ++j) pb[j] = B + min(n0 + 8 * j + r, (long long)g.N - 1) * g.sbn;
  double c[MB][NB][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) c[i][j][0] = c[i][j][1] = 0.0;
  constexpr int U = 4;   // steps whose operands are asked for together
  int k = 0;
  for (; k + 4 * U <= g.K; k += 4 * U) {
    double a[U][MB], b[U][NB];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long kk = k + 4 * u + q;
#pragma unroll
      for (int j = 0; j < NB; ++j) b[u][j] = __ldg(pb[j] + kk * g.sbk);
#pragma unroll
      for (int i = 0; i < MB; ++i) a[u][i] = __ldg(pa[i] + kk * g.sak);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < MB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) mma_f64(c[i][j], a[u][i], b[u][j]);
  }
  for (; k < g.K; k += 4) {
    const long long kk = k + q;
    const bool in = kk < g.K;   // beyond K: zeros
    double a[MB], b[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) b[j] = in ? __ldg(pb[j] + kk * g.sbk) : 0.0;
#pragma unroll
    for (int i = 0; i < MB; ++i) a[i] = in ? __ldg(pa[i] + kk * g.sak) : 0.0;
#pragma unroll
    for (int i = 0; i < MB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) mma_f64(c[i][j], a[i], b[j]);
  }
  double *C = g.C + blockIdx.z * g.zc;
#pragma unroll
  for (int i = 0; i < MB; ++i) {
    const int m = m0 + 8 * i + r;
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const long long n = n0 + 8 * j + 2 * q + e;
        if (n < g.N) C[m * g.scm + n * g.scn] = c[i][j][e];
      }
  }
}

}  // namespace

cudaError_t launch_dgemm(int M, int N, int K, const DMat &A, const DMat &B, double *C, long long scm, long long scn,
                         long long zc, int batch, cudaStream_t s) {
  if (M <= 0 || N <= 0 || batch <= 0) return cudaSuccess;
  if (K < 0 || batch > 65535) return cudaErrorInvalidValue;
  DGemmArgs g{M, N, K, A.p, B.p, C, A.rs, A.cs, B.rs, B.cs, scm, scn, A.z, B.z, zc};
  using Fn = void (*)(DGemmArgs);
  static const Fn fn[8] = {&dgemm_kernel<1, 2>, &dgemm_kernel<2, 2>, &dgemm_kernel<3, 2>, &dgemm_kernel<4, 2>,
                           &dgemm_kernel<5, 2>, &dgemm_kernel<6, 2>, &dgemm_kernel<7, 2>, &dgemm_kernel<8, 2>};
  // row chunks of at most 64, as even as they go; more and smaller ones while
  // the tiles would not fill the schedulers a few times over
  const int rows8 = (M + 7) / 8;
  const double cols = (double)((N + 15) / 16) * batch;
  int chunks = (rows8 + 7) / 8;
  while (chunks < rows8 && cols * chunks < 152 * 4 * 4) ++chunks;
  const int mb = (rows8 + chunks - 1) / chunks;
  chunks = (rows8 + mb - 1) / mb;
  if (chunks > 65535) return cudaErrorInvalidConfiguration;
  const long long tiles = ((long long)N + 15) / 16;
  const int warps = cols * chunks >= 152 * 4 * 4 ? 4 : 1;
  fn[mb - 1]<<<dim3((unsigned)((tiles + warps - 1) / warps), (unsigned)chunks, (unsigned)batch), 32 * warps, 0, s>>>(g);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace lgb
