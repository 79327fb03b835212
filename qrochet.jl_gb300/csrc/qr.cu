// Thin complex Householder QR (FP64) for canonize_site!(...; method=:qr) and for
// re-orthonormalising singular-vector blocks.
//
// Reflectors follow the published LAPACK zlarfg/zgeqr2/zung2r conventions (Householder vector
// with unit leading entry stored below the diagonal, beta real on the diagonal, H = I - tau v v^H,
// A <- H^H A during the factorisation, Q = H_0 H_1 ... H_{k-1} [I; 0]), so R has a real diagonal
// like the R that Julia's qr returns.
//
// Three schedules of the same factorisation:
//  - zqr_thin, up to 6144 rows: panels of 32 columns in one thread-block cluster each (house_panel_k), the
//    trailing columns and Q by products (zqr_thin_blocked).
//  - zqr_thin, more rows: the whole factorisation in one cooperative launch.  CTA b owns the columns
//    c = b (mod grid).  At step j every CTA reads column j (final after step j - 1), forms the
//    reflector's scalars itself (the same reduction order in every CTA gives the same bits), and
//    applies H_j^H to its own columns c > j; the owner of column j writes beta and the scaled
//    reflector into it at the start of step j + 1, once no CTA reads it any more.  One bounded grid
//    barrier per step.  Q needs no barrier at all: applying H_{k-1} .. H_0 to a column of [I; 0]
//    touches that column only, so each CTA runs all steps for its own columns in one launch.
//  - zqr_thin_steps: one reflector launch and one trailing-update launch per column (and one
//    Q launch per column), no scratch beyond tau; the allocation-free SVD uses it.
#include "kernels.cuh"
#include "prof.cuh"
#include "grid_sync.cuh"

namespace qr {

namespace {

constexpr int TPB = 256;
constexpr int QR_COOP_NT = 512;  // threads per CTA of the persistent factorisation

__device__ double block_sum_d(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < (blockDim.x >> 5)) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) red[0] = v;
  }
  __syncthreads();
  return red[0];
}

__device__ double2 block_sum_z(double2 v, double* red) {
  double re = block_sum_d(v.x, red);
  double im = block_sum_d(v.y, red);
  return make_double2(re, im);
}

// Householder reflector of x = A[j:m, j] (zlarfg).
__global__ void house_make_k(double2* A, int m, long lda, int j, double2* tau) {
  __shared__ double red[32];
  __shared__ double2 sh_scal;
  __shared__ int sh_skip;
  double2* x = A + j + (long)j * lda;
  const int len = m - j;
  double acc = 0.0;
  for (int t = 1 + threadIdx.x; t < len; t += blockDim.x) acc += x[t].x * x[t].x + x[t].y * x[t].y;
  double xnorm2 = block_sum_d(acc, red);
  if (threadIdx.x == 0) {
    double2 alpha = x[0];
    if (xnorm2 == 0.0 && alpha.y == 0.0) {
      tau[j] = make_double2(0.0, 0.0);
      sh_skip = 1;
    } else {
      double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2), alpha.x);
      tau[j] = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      double2 den = make_double2(alpha.x - beta, alpha.y);  // scal = 1 / (alpha - beta)
      double dd = den.x * den.x + den.y * den.y;
      sh_scal = make_double2(den.x / dd, -den.y / dd);
      x[0] = make_double2(beta, 0.0);
      sh_skip = 0;
    }
  }
  __syncthreads();
  if (sh_skip) return;
  double2 sc = sh_scal;
  for (int t = 1 + threadIdx.x; t < len; t += blockDim.x) x[t] = cmul(x[t], sc);
}

// A[j:m, c] <- (I - conj(tau_j) v v^H) A[j:m, c] for c in (j, n)   (H^H applied from the left)
__global__ void house_apply_left_k(double2* A, int m, int n, long lda, int j, const double2* tau) {
  __shared__ double red[32];
  const double2 t = tau[j];
  if (t.x == 0.0 && t.y == 0.0) return;
  const double2 tc = make_double2(t.x, -t.y);
  const double2* v = A + j + (long)j * lda;
  const int len = m - j;
  for (int c = j + 1 + blockIdx.x; c < n; c += gridDim.x) {
    double2* col = A + j + (long)c * lda;
    double2 acc = make_double2(0.0, 0.0);
    for (int r = threadIdx.x; r < len; r += blockDim.x) {
      double2 vr = (r == 0) ? make_double2(1.0, 0.0) : v[r];
      acc = cadd(acc, cmulc(vr, col[r]));
    }
    double2 w = cmul(tc, block_sum_z(acc, red));
    for (int r = threadIdx.x; r < len; r += blockDim.x) {
      double2 vr = (r == 0) ? make_double2(1.0, 0.0) : v[r];
      col[r] = csub(col[r], cmul(vr, w));
    }
    __syncthreads();
  }
}

// Q[j:m, c] <- (I - tau_j v v^H) Q[j:m, c] for c in [j, k)   (backward accumulation, zung2r)
__global__ void house_apply_q_k(double2* Q, int m, int k, long ldq, const double2* V, long ldv, int j,
                                const double2* tau) {
  __shared__ double red[32];
  const double2 t = tau[j];
  if (t.x == 0.0 && t.y == 0.0) return;
  const double2* v = V + j + (long)j * ldv;
  const int len = m - j;
  for (int c = j + blockIdx.x; c < k; c += gridDim.x) {
    double2* col = Q + j + (long)c * ldq;
    double2 acc = make_double2(0.0, 0.0);
    for (int r = threadIdx.x; r < len; r += blockDim.x) {
      double2 vr = (r == 0) ? make_double2(1.0, 0.0) : v[r];
      acc = cadd(acc, cmulc(vr, col[r]));
    }
    double2 w = cmul(t, block_sum_z(acc, red));
    for (int r = threadIdx.x; r < len; r += blockDim.x) {
      double2 vr = (r == 0) ? make_double2(1.0, 0.0) : v[r];
      col[r] = csub(col[r], cmul(vr, w));
    }
    __syncthreads();
  }
}

__global__ void extract_r_k(const double2* A, long lda, int k, int n, double2* R, long ldr) {
  long total = (long)k * n;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    long i = t % k, c = t / k;
    R[i + c * ldr] = (i <= c) ? A[i + c * lda] : make_double2(0.0, 0.0);
  }
}

// zlarfg scalars of x = A[j:m, j] (len = m - j), computed by every CTA alike (the same reduction
// order everywhere gives the same bits): tau = 0 (skip), or beta, tau and
// scal = 1 / (alpha - beta), through shared memory.
struct Reflector {
  double2 tau, scal;
  double beta;
  int skip;
};
__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ void reflector_of(const double2* x, int len, Reflector* out, double* red) {
  double acc = 0.0;
#pragma unroll 4
  for (int t = 1 + threadIdx.x; t < len; t += blockDim.x) acc += x[t].x * x[t].x + x[t].y * x[t].y;
  const double xnorm2 = block_sum_d(acc, red);
  {
    if (threadIdx.x == 0) {
      const double2 alpha = x[0];
      Reflector r;
      if (xnorm2 == 0.0 && alpha.y == 0.0) {
        r.tau = make_double2(0.0, 0.0);
        r.scal = make_double2(0.0, 0.0);
        r.beta = alpha.x;
        r.skip = 1;
      } else {
        const double beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2), alpha.x);
        r.tau = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
        const double2 den = make_double2(alpha.x - beta, alpha.y);
        const double dd = den.x * den.x + den.y * den.y;
        r.scal = make_double2(den.x / dd, -den.y / dd);
        r.beta = beta;
        r.skip = 0;
      }
      *out = r;
    }
  }
  __syncthreads();
}

// the pivot column j after its step: beta on the diagonal, the reflector scaled below it
__device__ void store_reflector(double2* x, int len, const Reflector& r) {
  if (r.skip) return;
  for (int t = 1 + threadIdx.x; t < len; t += blockDim.x) x[t] = cmul(x[t], r.scal);
  if (threadIdx.x == 0) x[0] = make_double2(r.beta, 0.0);
}

// One warp per owned column: col[0:len) -= v (conj(tau) v^H col), v = (1, x[1:] scal)
__global__ void __launch_bounds__(QR_COOP_NT) house_qr_coop_k(double2* A, int m, int n, long lda, double2* tau,
                                                               unsigned* bar) {
  __shared__ Reflector cur;
  __shared__ double red[32];
  Reflector prev;
  prev.skip = 1;
  const int k = m < n ? m : n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int G = (int)gridDim.x, b = (int)blockIdx.x;
  for (int j = 0; j < k; j++) {
    if (j > 0 && (j - 1) % G == b) store_reflector(A + (j - 1) + (long)(j - 1) * lda, m - (j - 1), prev);
    const double2* x = A + j + (long)j * lda;
    const int len = m - j;
    reflector_of(x, len, &cur, red);
    const Reflector r = cur;
    if (j % G == b) {
      if (threadIdx.x == 0) tau[j] = r.tau;
      prev = r;
    }
    if (!r.skip) {
      const double2 tc = make_double2(r.tau.x, -r.tau.y);
      const int c0 = j + 1 + ((b - (j + 1)) % G + G) % G;  // smallest owned column above j
      for (int c = c0 + warp * G; c < n; c += nw * G) {
        double2* col = A + j + (long)c * lda;
        double wr = 0.0, wi = 0.0;
#pragma unroll 8
        for (int t = lane; t < len; t += 32) {
          const double2 v = t == 0 ? make_double2(1.0, 0.0) : cmul(x[t], r.scal);
          const double2 y = col[t];
          wr += v.x * y.x + v.y * y.y;
          wi += v.x * y.y - v.y * y.x;
        }
        const double2 w = cmul(tc, make_double2(warp_sum_d(wr), warp_sum_d(wi)));
#pragma unroll 8
        for (int t = lane; t < len; t += 32) {
          const double2 v = t == 0 ? make_double2(1.0, 0.0) : cmul(x[t], r.scal);
          col[t] = csub(col[t], cmul(v, w));
        }
      }
    }
    if (!grid_barrier(bar)) return;
  }
  if (k > 0 && (k - 1) % G == b) store_reflector(A + (k - 1) + (long)(k - 1) * lda, m - (k - 1), prev);
}

// Q (m x k) = H_0 .. H_{k-1} [I; 0]: one CTA per column c, formed from e_c through H_c, ..., H_0
// (H_j touches rows j.. of the columns c >= j only, so columns need no synchronisation).  The
// longest columns (most reflectors) are dealt first.
__global__ void house_q_cols_k(double2* Q, int m, int k, long ldq, const double2* V, long ldv, const double2* tau) {
  __shared__ double red[32];
  for (int cc = blockIdx.x; cc < k; cc += gridDim.x) {
    const int c = k - 1 - cc;
    double2* col = Q + (long)c * ldq;
    for (int t = threadIdx.x; t < m; t += blockDim.x) col[t] = make_double2(t == c ? 1.0 : 0.0, 0.0);
    __syncthreads();
    for (int j = c; j >= 0; j--) {
      const double2 tj = tau[j];
      if (tj.x == 0.0 && tj.y == 0.0) continue;
      const double2* v = V + j + (long)j * ldv;
      const int len = m - j;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int t = threadIdx.x; t < len; t += blockDim.x) {
        const double2 vr = t == 0 ? make_double2(1.0, 0.0) : v[t];
        acc = cadd(acc, cmulc(vr, col[j + t]));
      }
      const double2 w = cmul(tj, block_sum_z(acc, red));
#pragma unroll 4
      for (int t = threadIdx.x; t < len; t += blockDim.x) {
        const double2 vr = t == 0 ? make_double2(1.0, 0.0) : v[t];
        col[j + t] = csub(col[j + t], cmul(vr, w));
      }
      __syncthreads();
    }
  }
}

// ---- blocked factorisation ---------------------------------------------------------------------
constexpr int QB = 32;            // panel columns
constexpr int QB_NT = 256;
constexpr int QB_LD = QB + 1;     // shared row stride (in complex numbers): column-wise fills hit all banks
constexpr int QB_CLUSTER = 16;
constexpr int QB_MAX_L = 384;     // rows a CTA holds (203 KB)

struct PanelShared {
  double2 part[QB_NT / 32][QB];          // a warp's sums
  double2 box[2][QB_CLUSTER][QB];        // every CTA's sums (by step parity)
  double2 sum4[4][QB];                   // partial sums over warps, then over CTAs
  double2 row[2][QB];                    // the pivot row
  double2 ws[QB], scal[QB], tau;
  double beta, ib;
  int skip;
};

__device__ __forceinline__ uint32_t qb_map(const void* p, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void qb_push(uint32_t addr, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void qb_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ double scale2(double y, int e) {  // y 2^e, the result normal
  return __longlong_as_double(__double_as_longlong(y) + ((long long)e << 52));
}
// 1 / x for 1e-300 < |x| < 1e300: Newton-Raphson in FP64 from an FP32 seed (2^-23 -> 2^-46 -> rounding).  The seed
// sees the fraction only, so no exponent of x leaves FP32's range.
__device__ __forceinline__ double inv_newton(double x) {
  const long long b = __double_as_longlong(x), e = (b >> 52) & 0x7ff;
  const double f = __longlong_as_double((b & 0x800fffffffffffffll) | (1023ll << 52));  // +-[1, 2)
  double y = (double)(1.f / (float)f);
  y = fma(y, fma(-f, y, 1.0), y);
  y = fma(y, fma(-f, y, 1.0), y);
  return scale2(y, (int)(1023 - e));
}
// 1 / sqrt(s), and sqrt(s) in *root, for 1e-280 < s < 1e280, in the same way
__device__ __forceinline__ double inv_root(double s, double* root) {
  const long long b = __double_as_longlong(s);
  const int h = (int)((b >> 52) - 1023) >> 1;  // s = f 4^h, f in [1, 4)
  const double f = __longlong_as_double(b - ((long long)(2 * h) << 52));
  double y = (double)rsqrtf((float)f);
  y = fma(0.5 * y, fma(-f * y, y, 1.0), y);
  y = fma(0.5 * y, fma(-f * y, y, 1.0), y);
  double r = f * y;
  r = fma(0.5 * y, fma(-r, r, f), r);
  *root = scale2(r, h);
  return scale2(y, -h);
}

// Householder panel A[0:m, 0:nb] (nb <= QB) in one cluster of cs CTAs, CTA r holding rows r L .. r L + L - 1
// in shared memory, row by row.  Step j needs one exchange: with d_c = sum over rows > j of conj(x) a_c for
// the pivot column x and every column c (d_j = |x|^2) and the pivot row, every CTA knows beta, tau and
// v^H a_c = a_jc + conj(scal) d_c, v = (1, x scal), and updates its rows.  Lanes are columns, and once fewer
// than 16 (8) are left a warp takes 2 (4) rows at a time.  On exit R's rows are in A, the unit lower
// trapezoid (zeros above the diagonal) in V (m x nb), and tau.
// Bound: at 16 rows a CTA the latency of a step (~5 us: a 16-CTA exchange 1.1, sums 0.9, the reflector's serial
// FP64 chain 2); at 64 rows and more the FP64 pipe (8 FMAs per element and step, 2 per cycle and SM): a panel of
// 1024 rows takes 247 us with that pipe 57% active.
__global__ void __launch_bounds__(QB_NT) house_panel_k(double2* __restrict__ A, long lda, int m, int nb,
                                                       double2* __restrict__ V, long ldv, double2* __restrict__ tau, int L,
                                                       int cs) {
  extern __shared__ __align__(16) double2 qb_rows[];
  __shared__ PanelShared sh;
  const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = rank * L, rows = max(0, min(L, m - r0));
  for (int e = tid; e < L * QB; e += QB_NT) {
    const int r = e % L, c = e / L;
    qb_rows[r * QB_LD + c] = (r < rows && c < nb) ? A[r0 + r + (long)c * lda] : make_double2(0.0, 0.0);
  }
  __syncwarp();
  qb_cluster_sync();
  const int steps = min(nb, m);
  for (int j = 0; j < steps; j++) {
    const int par = j & 1;
    const int wd = j < 16 ? 32 : j < 24 ? 16 : 8;  // columns a row takes: c0 .. 31
    const int c0 = 32 - wd, per = 32 / wd, c = c0 + lane % wd, sub = lane / wd;
    const int first = max(0, j + 1 - r0);          // local rows below the pivot
    // four independent sums: an FP64 addition's latency is longer than a row's loads
    double2 acc = make_double2(0.0, 0.0), ac2 = acc;
#pragma unroll 2
    for (int r = first + warp * per + sub; r < rows; r += (QB_NT / 32) * per) {
      const double2 x = qb_rows[r * QB_LD + j], a = qb_rows[r * QB_LD + c];
      acc.x += x.x * a.x;
      ac2.x += x.y * a.y;
      acc.y += x.x * a.y;
      ac2.y -= x.y * a.x;
    }
    acc = cadd(acc, ac2);
    for (int o = wd; o < 32; o <<= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (sub == 0) sh.part[warp][c] = acc;
    __syncthreads();
    // sums over warps, and below over CTAs, in two stages spread over the warps: a warp-wide FP64
    // instruction occupies its scheduler's pipe for 64 cycles, so one warp adding alone took 1100 and 2500
    if (warp < 4) sh.sum4[warp][lane] = cadd(sh.part[2 * warp][lane], sh.part[2 * warp + 1][lane]);
    __syncthreads();
    if (warp < 2) {  // real parts, imaginary parts
      const double* v = &sh.sum4[0][0].x + warp;
      (&sh.part[0][0].x)[2 * lane + warp] = (v[2 * lane] + v[2 * (QB + lane)]) + (v[2 * (2 * QB + lane)] + v[2 * (3 * QB + lane)]);
    }
    __syncthreads();
    for (int e = tid; e < cs * QB; e += QB_NT) {
      const int to = e / QB, cc = e % QB;
      if (cc >= c0) qb_push(qb_map(&sh.box[par][rank][cc], to), sh.part[0][cc]);
      if (j >= r0 && j < r0 + L && cc >= c0) qb_push(qb_map(&sh.row[par][cc], to), qb_rows[(j - r0) * QB_LD + cc]);
    }
    __syncwarp();
    qb_cluster_sync();
    {
      const int grp = warp >> 1, re = warp & 1;  // four groups of up to four CTAs, real or imaginary parts
      const double* b = &sh.box[par][0][0].x + 2 * lane + re;
      double v = 0.0;
      if (lane >= c0 && grp < cs) {
        v = b[2 * QB * grp];
        if (grp + 4 < cs) v += b[2 * QB * (grp + 4)];
        if (grp + 8 < cs) v += b[2 * QB * (grp + 8)] + b[2 * QB * (grp + 12)];
      }
      (&sh.sum4[grp][lane].x)[re] = v;
    }
    __syncthreads();
    if (warp == 0) {
      double2 d = sh.sum4[0][lane];
      if (cs > 1) d = cadd(d, sh.sum4[1][lane]);
      if (cs > 2) d = cadd(d, cadd(sh.sum4[2][lane], sh.sum4[3][lane]));
      const double2 a = sh.row[par][lane];
      if (lane == j) {
        if (d.x == 0.0 && a.y == 0.0) {
          sh.tau = sh.scal[j] = make_double2(0.0, 0.0);
          sh.beta = a.x;
          sh.ib = 0.0;
          sh.skip = 1;
        } else {
          // one root and one reciprocal, by Newton steps
          const double s2 = a.x * a.x + a.y * a.y + d.x;
          const bool neg = signbit(a.x);
          double beta, ib, idd;
          if (s2 > 1e-280 && s2 < 1e280) {
            double nrm;
            const double inr = inv_root(s2, &nrm);
            beta = neg ? nrm : -nrm;
            ib = neg ? inr : -inr;
            const double dx = a.x - beta;
            idd = inv_newton(dx * dx + a.y * a.y);
          } else {
            beta = -copysign(sqrt(s2), a.x);
            ib = 1.0 / beta;
            const double dx = a.x - beta;
            idd = 1.0 / (dx * dx + a.y * a.y);
          }
          const double2 den = make_double2(a.x - beta, a.y);
          sh.tau = make_double2(-den.x * ib, -a.y * ib);
          sh.scal[j] = make_double2(den.x * idd, -den.y * idd);
          sh.beta = beta;
          sh.ib = ib;
          sh.skip = 0;
        }
      }
      __syncwarp();
      const double2 sc = sh.scal[j], t = sh.tau;
      // w_c = v^H a_c conj(tau) = conj(tau) a_jc - d_c / beta (conj(tau) conj(scal) = -1 / beta);
      // a -= x (scal w_c).  The pivot column stays unscaled here
      const double2 ta = cmulc(t, a);
      const double ib = sh.ib;
      const double2 w = make_double2(fma(-ib, d.x, ta.x), fma(-ib, d.y, ta.y));
      sh.ws[lane] = cmul(sc, w);
      if (!sh.skip && j >= r0 && j < r0 + L && lane >= j)
        qb_rows[(j - r0) * QB_LD + lane] = lane == j ? make_double2(sh.beta, 0.0) : csub(a, w);
      if (lane == 0 && rank == 0) tau[j] = t;
    }
    __syncthreads();
    if (!sh.skip && c > j) {
      const double2 ws = sh.ws[c];
      for (int r = first + warp * per + sub; r < rows; r += (QB_NT / 32) * per) {
        const double2 x = qb_rows[r * QB_LD + j];
        double2 a = qb_rows[r * QB_LD + c];
        a.x -= x.x * ws.x - x.y * ws.y;
        a.y -= x.x * ws.y + x.y * ws.x;
        qb_rows[r * QB_LD + c] = a;
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < L * QB; e += QB_NT) {
    const int r = e % L, c = e / L, g = r0 + r;
    if (r >= rows || c >= nb) continue;
    const double2 v = qb_rows[r * QB_LD + c];
    if (g <= c) A[g + (long)c * lda] = v;
    V[g + (long)c * ldv] = g > c ? cmul(v, sh.scal[c]) : make_double2(g == c ? 1.0 : 0.0, 0.0);
  }
  __syncwarp();
  qb_cluster_sync();  // no CTA leaves while another may still push into it
}

// W (nb x nc, ld QB) <- T^H W (adjoint) or T W, T the triangular factor of the panel's block reflector.  With
// S = V^H V its inverse is known, T^-1 = diag(1 / tau) + strictly upper part of S, so T is never formed: a
// warp per column substitutes forwards (T^H) or backwards (T), lane i holding entry i.
__global__ void __launch_bounds__(128) wy_solve_k(const double2* __restrict__ S, const double2* __restrict__ tau, int nb,
                                                  double2* __restrict__ W, int nc, int adjoint) {
  __shared__ double2 sS[QB][QB + 1], st[QB];
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) sS[e % nb][e / nb] = S[e % nb + (long)(e / nb) * QB];
  if (threadIdx.x < nb) st[threadIdx.x] = tau[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31, c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= nc) return;
  double2 w = lane < nb ? W[lane + (long)c * QB] : make_double2(0.0, 0.0);
  for (int u = 0; u < nb; u++) {
    const int j = adjoint ? u : nb - 1 - u;
    const double2 t = st[j];
    double2 x = lane == j ? (adjoint ? cmulc(t, w) : cmul(t, w)) : w;  // conj(tau) w or tau w
    x.x = __shfl_sync(0xffffffffu, x.x, j);
    x.y = __shfl_sync(0xffffffffu, x.y, j);
    if (lane == j) w = x;
    else if (adjoint ? (lane > j && lane < nb) : lane < j)
      w = csub(w, adjoint ? cmulc(sS[j][lane], x) : cmul(sS[lane][j], x));
  }
  if (lane < nb) W[lane + (long)c * QB] = w;
}

inline int cuda_ok_qr(cudaError_t e) { return e == cudaSuccess ? QR_OK : cuda_fail(e, "Householder QR"); }

inline unsigned cols_grid(int ncols) {
  int g = ncols < 1 ? 1 : ncols;
  return (unsigned)(g > 152 * 8 ? 152 * 8 : g);
}

}  // namespace

int zqr_thin_steps(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
                   long ldr, double2* tau) {
  if (m <= 0 || n <= 0) return QR_OK;
  const int k = m < n ? m : n;
  for (int j = 0; j < k; j++) {
    house_make_k<<<1, TPB, 0, s>>>(A, m, lda, j, tau);
    QR_CHECK_LAUNCH("house_make_k");
    if (j + 1 < n) {
      house_apply_left_k<<<cols_grid(n - j - 1), TPB, 0, s>>>(A, m, n, lda, j, tau);
      QR_CHECK_LAUNCH("house_apply_left_k");
    }
  }
  if (R) {
    long total = (long)k * n;
    unsigned g = (unsigned)((total + TPB - 1) / TPB);
    extract_r_k<<<g > 4864 ? 4864 : g, TPB, 0, s>>>(A, lda, k, n, R, ldr);
    QR_CHECK_LAUNCH("extract_r_k");
  }
  if (Q) {
    QR_TRY(zset_identity(s, Q, m, k, ldq));
    for (int j = k - 1; j >= 0; j--) {
      house_apply_q_k<<<cols_grid(k - j), TPB, 0, s>>>(Q, m, k, ldq, A, lda, j, tau);
      QR_CHECK_LAUNCH("house_apply_q_k");
    }
  }
  return QR_OK;
}

static int zqr_thin_coop(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
                         long ldr, double2* tau, int sms);
static int zqr_thin_blocked(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
                            long ldr, double2* tau);

int zqr_thin(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
             long ldr, double2* tau) {
  if (m <= 0 || n <= 0) return QR_OK;
  int sms = 0, per_sm = 0;
  QR_TRY(device_sm_count(&sms));
  QR_TRY(blocks_per_sm((const void*)house_qr_coop_k, QR_COOP_NT, 0, &per_sm));
  if (per_sm < 1) return zqr_thin_steps(s, A, m, n, lda, Q, ldq, R, ldr, tau);
  // complex flops: factorisation 8 (m n^2 - n^3 / 3), the same again to form Q
  const double fl = 8.0 * ((double)m * n * n - (double)n * n * n / 3.0) * (Q ? 2.0 : 1.0);
  const int pr = prof_begin(s, PK_QR, fl, 16.0 * (double)m * n * (Q ? 3.0 : 2.0));
  const int rc0 = m <= QB_CLUSTER * QB_MAX_L ? zqr_thin_blocked(s, A, m, n, lda, Q, ldq, R, ldr, tau)
                                             : zqr_thin_coop(s, A, m, n, lda, Q, ldq, R, ldr, tau, sms);
  prof_end(s, pr);
  return rc0;
}

// the cooperative factorisation, R and Q of zqr_thin
static int zqr_thin_coop(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
                         long ldr, double2* tau, int sms) {
  const int k = m < n ? m : n;
  // one 512-thread CTA per SM, one warp per owned column: a step is the reflector (warp 0 of every
  // CTA), the column updates of the CTA's warps in parallel, and the grid barrier
  int grid = std::min(sms, std::max(1, n - 1));
  unsigned* bar = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&bar, 4 * sizeof(unsigned), s);
  if (e != cudaSuccess) return fail(QR_ENOMEM, std::string("QR barrier: ") + cudaGetErrorString(e));
  int rc = cuda_ok_qr(cudaMemsetAsync(bar, 0, 4 * sizeof(unsigned), s));
  if (!rc) {
    double2* Ap = A;
    int mm = m, nn = n;
    long ld = lda;
    double2* tp = tau;
    unsigned* bp = bar;
    void* args[] = {&Ap, &mm, &nn, &ld, &tp, &bp};
    rc = cuda_ok_qr(cudaLaunchCooperativeKernel((const void*)house_qr_coop_k, dim3(grid), dim3(QR_COOP_NT), args, 0, s));
    count_launch();
  }
  unsigned hb[3] = {0, 0, 0};
  if (!rc) rc = cuda_ok_qr(cudaMemcpyAsync(hb, bar, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  if (!rc) rc = cuda_ok_qr(cudaStreamSynchronize(s));
  cudaFreeAsync(bar, s);
  if (rc) return rc;
  if (hb[2]) return fail(QR_ECUDA, "Householder QR: a grid barrier timed out");
  if (R) {
    long total = (long)k * n;
    unsigned g = (unsigned)((total + TPB - 1) / TPB);
    extract_r_k<<<g > 4864 ? 4864 : g, TPB, 0, s>>>(A, lda, k, n, R, ldr);
    QR_CHECK_LAUNCH("extract_r_k");
  }
  if (Q) {
    house_q_cols_k<<<cols_grid(k), TPB, 0, s>>>(Q, m, k, ldq, A, lda, tau);
    QR_CHECK_LAUNCH("house_q_cols_k");
  }
  return QR_OK;
}

// 1024 x 512 with Q: 7.7 ms (the column-at-a-time cooperative kernel and Q kernel: 17.8), 2048 x 1024 23.8 (84),
// 2048 x 2048 49.7 (220), 256 x 256 2.3 (3.5).  Panels of QB columns by house_panel_k; the block reflectors I - V T V^H are applied to the trailing columns
// and to [I; 0] as products (W = V^H C, W <- T^H W, C -= V W).
static int zqr_thin_blocked(cudaStream_t s, double2* A, int m, int n, long lda, double2* Q, long ldq, double2* R,
                            long ldr, double2* tau) {
  const int k = m < n ? m : n, np = (k + QB - 1) / QB;
  const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
  double2* ws = nullptr;
  const size_t nv = (size_t)m * k, nw = (size_t)QB * std::max(n, k), ns = (size_t)QB * QB * np;
  cudaError_t e = cudaMallocAsync((void**)&ws, sizeof(double2) * (nv + nw + ns), s);
  if (e != cudaSuccess) return fail(QR_ENOMEM, std::string("QR reflectors: ") + cudaGetErrorString(e));
  double2 *V = ws, *W = V + nv, *S = W + nw;
  // C (rows p0.. of m, nc columns) <- (I - V_p op(T) V_p^H) C
  auto apply = [&](int p, double2* C, long ldc, int nc, int adjoint) -> int {
    const int p0 = p * QB, nb = std::min(QB, k - p0), mj = m - p0;
    const double2* Vp = V + p0 + (long)p0 * m;
    // the unit triangle apart: beside its ones the sliced product would round the long, small part of V
    // relative to 1 (2048 rows: 8x the error of an FP64 product)
    const int lo = mj - nb;
    if (lo > 0) QR_TRY(zgemm(s, OP_C, OP_N, nb, nc, lo, one, Vp + nb, m, 0, C + nb, ldc, 0, zero, W, QB, 0, 1, nullptr,
                             true));
    QR_TRY(zgemm_spread(s, OP_C, OP_N, nb, nc, nb, one, Vp, m, 0, C, ldc, 0, lo > 0 ? one : zero, W, QB, 0, 1, nullptr));
    wy_solve_k<<<ceil_div(nc, 4), 128, 0, s>>>(S + (size_t)QB * QB * p, tau + p0, nb, W, nc, adjoint);
    QR_CHECK_LAUNCH("wy_solve_k");
    QR_TRY(zgemm_spread(s, OP_N, OP_N, nb, nc, nb, make_double2(-1.0, 0.0), Vp, m, 0, W, QB, 0, one, C, ldc, 0, 1, nullptr));
    return zgemm_sub(s, lo, nc, nb, Vp + nb, m, W, QB, C + nb, ldc);
  };
  auto run = [&]() -> int {
    QR_TRY(set_func_attr_once((const void*)house_panel_k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    QR_TRY(set_func_attr_once((const void*)house_panel_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              QB_MAX_L * QB_LD * (int)sizeof(double2)));
    for (int p = 0; p < np; p++) {
      const int p0 = p * QB, nb = std::min(QB, k - p0), mj = m - p0;
      // at least 16 rows per CTA: below that the exchange costs more than the rows
      int cs = 1;
      while (cs < QB_CLUSTER && mj > 16 * cs) cs *= 2;
      const int L = (mj + cs - 1) / cs;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(cs);
      cfg.blockDim = dim3(QB_NT);
      cfg.dynamicSmemBytes = (size_t)L * QB_LD * sizeof(double2);
      cfg.stream = s;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = cs;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      double2* Vp = V + p0 + (long)p0 * m;
      QR_CUDA(cudaLaunchKernelEx(&cfg, house_panel_k, A + p0 + (long)p0 * lda, lda, mj, nb, Vp, (long)m, tau + p0, L, cs));
      count_launch();
      const int nc = n - p0 - nb;
      if (nc > 0 || Q) QR_TRY(zherk_spread(s, nb, mj, Vp, m, S + (size_t)QB * QB * p, QB));
      if (nc > 0) QR_TRY(apply(p, A + p0 + (long)(p0 + nb) * lda, lda, nc, 1));
    }
    if (R) {
      const long total = (long)k * n;
      extract_r_k<<<(unsigned)std::min<long>((total + TPB - 1) / TPB, 4864), TPB, 0, s>>>(A, lda, k, n, R, ldr);
      QR_CHECK_LAUNCH("extract_r_k");
    }
    if (Q) {
      QR_TRY(zset_identity(s, Q, m, k, ldq));
      for (int p = np - 1; p >= 0; p--) QR_TRY(apply(p, Q + p * QB + (long)(p * QB) * ldq, ldq, k - p * QB, 0));
    }
    return QR_OK;
  };
  const int rc = run();
  cudaFreeAsync(ws, s);
  return rc;
}

}  // namespace qr
