// Complex FP64 GEMM, C[b] = alpha op(A[b]) diag(dk) op(B[b]) + beta C[b]:
//   op: N (as stored, column-major), T (transpose), C (conjugate transpose), R (conjugate).
//
// Two kernels.  Products from OZ_MIN_WORK multiply-adds on (alpha = 1, beta = 0: every call of the
// library) run on the tensor cores as exact integer slices (gemm_oz.cu).  The rest run here, in FP64:
// an SM does 7 GFLOP/s in FP64 whatever instruction issues it (DMMA or DFMA), so a small product is fast
// only when all SMs share it.  zgemm_spread_k gives a CTA 32 elements of C and a warp a slice of K.
#include "kernels.cuh"
#include "prof.cuh"

namespace qr {

namespace {

struct Strided {
  const double2* p;
  long s0, sk, sb;  // strides along the outer index, along K, and between batch entries
  int conj;
};

__global__ void __launch_bounds__(256) zgemm_spread_k(const Strided a, const Strided b, int M, int N, int K,
                                                      double2 alpha, double2 beta, double2* __restrict__ C, long ldc,
                                                      long sC, const double* __restrict__ dk) {
  __shared__ double2 part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const long e = blockIdx.x * 32L + lane;
  const bool in = e < (long)M * N;
  const int i = in ? (int)(e % M) : 0, j = in ? (int)(e / M) : 0;
  const double2* pa = a.p + blockIdx.z * a.sb + i * a.s0;
  const double2* pb = b.p + blockIdx.z * b.sb + j * b.s0;
  // conjugation flips a sign bit on the integer pipe: an FP64 multiply costs as much as an FMA here
  const long long ca = a.conj ? 1ll << 63 : 0, cb = b.conj ? 1ll << 63 : 0;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int k = warp; k < K; k += nw) {
    double2 x = pa[k * a.sk], y = pb[k * b.sk];
    if (dk) x = cscale(x, dk[k]);
    x.y = __longlong_as_double(__double_as_longlong(x.y) ^ ca);
    y.y = __longlong_as_double(__double_as_longlong(y.y) ^ cb);
    acc.x += x.x * y.x - x.y * y.y;
    acc.y += x.x * y.y + x.y * y.x;
  }
  part[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && in) {
    for (int w = 1; w < nw; w++) acc = cadd(acc, part[w][lane]);
    double2* c = C + blockIdx.z * sC + i + (long)j * ldc;
    acc = cmul(alpha, acc);
    if (beta.x != 0.0 || beta.y != 0.0) acc = cadd(acc, cmul(beta, *c));
    *c = acc;
  }
}

// From this many complex multiply-adds on, the three launches of the sliced product cost less than the
// spread kernel's FP64 time (4 DFMA each at 2 per SM and cycle): 96 x 128 x 96 takes 25 us sliced and 19
// here, 128 x 128 x 128 25 and 31, 256 x 512 x 256 34 and 372.  (The 64 x 64-tile DMMA kernel that ran all
// sizes before took 592 us at 128^3, 1176 at 256 x 512 x 256 and 64.9 ms at 2048^3; sliced: 2.07 ms.)
constexpr double OZ_MIN_WORK = 1.5 * (1 << 20);

}  // namespace

int zgemm_spread(cudaStream_t s, int opA, int opB, int M, int N, int K, double2 alpha, const double2* A, long lda,
                 long sA, const double2* B, long ldb, long sB, double2 beta, double2* C, long ldc, long sC, int batch,
                 const double* dk) {
  if (M <= 0 || N <= 0 || batch <= 0) return QR_OK;
  if (K <= 0) return zscale_matrix(s, M, N, beta, C, ldc, sC, batch);  // C = beta * C
  const bool an = opA == OP_N || opA == OP_R, bn = opB == OP_N || opB == OP_R;
  const Strided a = {A, an ? 1 : lda, an ? lda : 1, sA, opA == OP_C || opA == OP_R};
  const Strided b = {B, bn ? ldb : 1, bn ? 1 : ldb, sB, opB == OP_C || opB == OP_R};
  const int warps = K >= 32 ? 8 : K >= 8 ? 4 : 1;
  zgemm_spread_k<<<dim3(ceil_div((long)M * N, 32), 1, batch), 32 * warps, 0, s>>>(a, b, M, N, K, alpha, beta, C, ldc, sC, dk);
  QR_CHECK_LAUNCH("zgemm_spread_k");
  return QR_OK;
}

int zgemm(cudaStream_t s, int opA, int opB, int M, int N, int K, double2 alpha,
          const double2* A, long lda, long sA, const double2* B, long ldb, long sB,
          double2 beta, double2* C, long ldc, long sC, int batch, const double* dk) {
  if (M <= 0 || N <= 0 || batch <= 0) return QR_OK;
  if (opA < 0 || opA > 3 || opB < 0 || opB > 3) return fail(QR_EINVAL, "zgemm: bad op");
  const double work = (double)M * N * K * batch;
  const double by = 16.0 * ((double)M * K + (double)K * N + 2.0 * M * N) * batch;
  const int pr = prof_begin(s, PK_ZGEMM, 8.0 * work, by);
  const bool plain = alpha.x == 1.0 && alpha.y == 0.0 && beta.x == 0.0 && beta.y == 0.0;
  const int rc = plain && work >= OZ_MIN_WORK && zgemm_oz_fits(M, N, K)
                     ? zgemm_oz(s, opA, opB, M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, dk)
                     : zgemm_spread(s, opA, opB, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, dk);
  prof_end(s, pr);
  return rc;
}

}  // namespace qr
