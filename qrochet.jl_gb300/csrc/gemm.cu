// Complex FP64 GEMM, C[b] = alpha op(A[b]) diag(dk) op(B[b]) + beta C[b]:
//   op: N (as stored, column-major), T (transpose), C (conjugate transpose), R (conjugate).
//
// Two kernels.  Products from OZ_MIN_WORK multiply-adds on (alpha = 1, beta = 0: every large product of the
// library) run on the tensor cores as integer slices (gemm_oz.cu).  The rest run here, in FP64:
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

// OUT elements of C per CTA; a warp's lanes are OUT elements x 32 / OUT slices of K, its warps split K
// further.  OUT = 8 for products of few elements (a panel's 32 x 32 Gram matrix over 1024 rows: 128 CTAs).
template <int OUT>
__global__ void __launch_bounds__(256) zgemm_spread_k(const Strided a, const Strided b, int M, int N, int K,
                                                      double2 alpha, double2 beta, double2* __restrict__ C, long ldc,
                                                      long sC, const double* __restrict__ dk, int herm) {
  __shared__ double2 part[8][OUT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int el = lane % OUT, ks = lane / OUT;
  const long e = blockIdx.x * (long)OUT + el;
  bool in = e < (long)M * N;
  int i = in ? (int)(e % M) : 0, j = in ? (int)(e / M) : 0;
  if (herm && in) {  // e counts the M (M + 1) / 2 entries on and above the diagonal, by columns
    j = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
    while ((long)j * (j + 1) / 2 > e) j--;
    while ((long)(j + 1) * (j + 2) / 2 <= e) j++;
    i = (int)(e - (long)j * (j + 1) / 2);
    in = j < N;
    if (!in) i = j = 0;
  }
  const double2* pa = a.p + blockIdx.z * a.sb + i * a.s0;
  const double2* pb = b.p + blockIdx.z * b.sb + j * b.s0;
  // conjugation flips a sign bit on the integer pipe: an FP64 multiply costs as much as an FMA here
  const long long ca = a.conj ? 1ll << 63 : 0, cb = b.conj ? 1ll << 63 : 0;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int k = warp * (32 / OUT) + ks; k < K; k += nw * (32 / OUT)) {
    double2 x = pa[k * a.sk], y = pb[k * b.sk];
    if (dk) x = cscale(x, dk[k]);
    x.y = __longlong_as_double(__double_as_longlong(x.y) ^ ca);
    y.y = __longlong_as_double(__double_as_longlong(y.y) ^ cb);
    acc.x += x.x * y.x - x.y * y.y;
    acc.y += x.x * y.y + x.y * y.x;
  }
  for (int o = OUT; o < 32; o <<= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if (ks == 0) part[warp][el] = acc;
  __syncthreads();
  if (warp == 0 && ks == 0 && in) {
    for (int w = 1; w < nw; w++) acc = cadd(acc, part[w][el]);
    double2* c = C + blockIdx.z * sC + i + (long)j * ldc;
    acc = cmul(alpha, acc);
    if (beta.x != 0.0 || beta.y != 0.0) acc = cadd(acc, cmul(beta, *c));
    *c = acc;
    if (herm && i != j) C[j + (long)i * ldc] = cconj(acc);
  }
}

}  // namespace

int zgemm_spread(cudaStream_t s, int opA, int opB, int M, int N, int K, double2 alpha, const double2* A, long lda,
                 long sA, const double2* B, long ldb, long sB, double2 beta, double2* C, long ldc, long sC, int batch,
                 const double* dk) {
  if (M <= 0 || N <= 0 || batch <= 0) return QR_OK;
  if (K <= 0) return zscale_matrix(s, M, N, beta, C, ldc, sC, batch);  // C = beta * C
  const bool an = opA == OP_N || opA == OP_R, bn = opB == OP_N || opB == OP_R;
  const Strided a = {A, an ? 1 : lda, an ? lda : 1, sA, opA == OP_C || opA == OP_R};
  const Strided b = {B, bn ? ldb : 1, bn ? 1 : ldb, sB, opB == OP_C || opB == OP_R};
  const bool few = (long)M * N * batch < 32 * 76;  // 32 elements a CTA would reach less than half of the 152 SMs
  const int slices = few ? 4 : 1, warps = K >= 32 * slices ? 8 : K >= 8 * slices ? 4 : 1;
  const dim3 grid(ceil_div((long)M * N, few ? 8 : 32), 1, batch);
  if (few) zgemm_spread_k<8><<<grid, 32 * warps, 0, s>>>(a, b, M, N, K, alpha, beta, C, ldc, sC, dk, 0);
  else zgemm_spread_k<32><<<grid, 32 * warps, 0, s>>>(a, b, M, N, K, alpha, beta, C, ldc, sC, dk, 0);
  QR_CHECK_LAUNCH("zgemm_spread_k");
  return QR_OK;
}

int zherk_spread(cudaStream_t s, int n, int K, const double2* A, long lda, double2* C, long ldc) {
  if (n <= 0) return QR_OK;
  const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
  if (K <= 0) return zscale_matrix(s, n, n, zero, C, ldc, 0, 1);
  const Strided a = {A, lda, 1, 0, 1}, b = {A, lda, 1, 0, 0};
  const long total = (long)n * (n + 1) / 2;
  const bool few = total < 32 * 76;  // as in zgemm_spread
  const int slices = few ? 4 : 1, warps = K >= 32 * slices ? 8 : K >= 8 * slices ? 4 : 1;
  const unsigned grid = ceil_div(total, few ? 8 : 32);
  if (few) zgemm_spread_k<8><<<grid, 32 * warps, 0, s>>>(a, b, n, n, K, one, zero, C, ldc, 0, nullptr, 1);
  else zgemm_spread_k<32><<<grid, 32 * warps, 0, s>>>(a, b, n, n, K, one, zero, C, ldc, 0, nullptr, 1);
  QR_CHECK_LAUNCH("zgemm_spread_k");
  return QR_OK;
}

int zgemm(cudaStream_t s, int opA, int opB, int M, int N, int K, double2 alpha,
          const double2* A, long lda, long sA, const double2* B, long ldb, long sB,
          double2 beta, double2* C, long ldc, long sC, int batch, const double* dk, bool normwise) {
  if (M <= 0 || N <= 0 || batch <= 0) return QR_OK;
  if (opA < 0 || opA > 3 || opB < 0 || opB > 3) return fail(QR_EINVAL, "zgemm: bad op");
  const double work = (double)M * N * K * batch;
  const double by = 16.0 * ((double)M * K + (double)K * N + 2.0 * M * N) * batch;
  const int pr = prof_begin(s, PK_ZGEMM, 8.0 * work, by);
  const bool plain = alpha.x == 1.0 && alpha.y == 0.0 && beta.x == 0.0 && beta.y == 0.0;
  const int rc = plain && work >= OZ_MIN_WORK && zgemm_oz_fits(M, N, K)
                     ? zgemm_oz(s, opA, opB, M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, dk, !normwise)
                     : zgemm_spread(s, opA, opB, M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, dk);
  prof_end(s, pr);
  return rc;
}

}  // namespace qr
