// Batched engine: many independent chains of uneven length and bond dimension evolved together,
// one fused launch per brick-wall layer, the whole circuit captured in one CUDA graph.
//
// The work unit is evolve_2site! + truncate! (Chain.jl:606-661, 390-422) on |0...0> chains
// (convert(Chain, zeros(Product, n)), Chain.jl:174-183), then expect of Pauli strings
// (Chain.jl:724-735).  Everything a layer needs stays on the device:
//   - every chain's sites live in fixed-capacity buffers: bond b of an n-qubit chain can never
//     exceed cap_b = min(chi_max, 2^min(b+1, n-b-1)), so site i is allocated as
//     cap_{i-1} x 2 x cap_i and holds its current (chi_l, 2, chi_r) array densely;
//   - bond dimensions, Lambda flags and Lambda vectors are device arrays that the kernels read
//     and rewrite: the truncation decision (the first min(k, maxdim) singular values above the
//     threshold) is taken on the device, so no layer waits for the host;
//   - one cluster of 1, 4 or 8 CTAs runs one whole gate step: theta = A_l diag(Lambda) A_r, the
//     gate, a Jacobi SVD (theta of at most 128 x 128: chi_max <= 64; FP32 sweeps first above 8
//     columns, the finish in FP64 or, with QR_MIXED above 32 columns, in double-float on the FP32
//     pipes), the sort, the truncation, re-orthonormalisation of the kept vectors when their
//     singular values fall below 1e-3 sigma_max (classical Gram-Schmidt twice), and the write-back
//     of U, Vh and Lambda.  A layer's gates sit on disjoint bonds, so the clusters of one launch
//     never touch the same site;
//   - the expectation values are one more launch: one cluster per Pauli string sweeps the chain's
//     environment (FP64).
// The layer kernel's CTA size comes from a small autotuner (timed on synthetic gate steps of the
// batch's largest bond class, cached per device and class, optionally in a file).
#include <vector>
#include <mutex>
#include <map>
#include <string>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <algorithm>
#include "kernels.cuh"
#include "jacobi_df.cuh"
#include "team_svd.cuh"

namespace qr {
namespace {

constexpr int BT_MAXK = 128;         // largest theta side: chi_max <= 64
constexpr int BT_MAXCHI = BT_MAXK / 2;
constexpr int BT_MAX_SWEEPS = 60;
// workspace of a gate step of theta up to side x side (double2): theta, B, V and the kept vectors, the SVD's
// own, a column of coefficients and one of norms
constexpr size_t slot_size(int side) { return 4 * (size_t)side * side + team_ws(side) + 2 * BT_MAXK; }
constexpr int BT_PRE_MIN = 8;   // the SVD sweeps in FP32 first above this many columns
constexpr int BT_TEAM_MAX = 32;  // and its FP64 refinement by products pays up to this many
constexpr int BT_MAXTEAM = 8;    // CTAs per gate step

__device__ __forceinline__ void cfma(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}

struct BTask {
  double2* sl;          // left site buffer
  double2* sr;          // right site buffer
  double* lam;          // Lambda buffer of the bond
  int* bd;              // bond dimensions of the chain
  int* haslam;          // Lambda flags of the chain
  const double2* gate;  // 4 x 4 row-major, [(o1',o2'),(o1,o2)]
  int* status;          // the request's status word
  double threshold;
  int bond, nb, maxdim, pad;
};

struct BObs {
  double2* const* sites;  // n site pointers
  double* const* lams;    // n-1 Lambda pointers
  const int* bd;
  const int* haslam;
  const int* pauli;  // per site 0 I, 1 X, 2 Y, 3 Z
  double2* out;
  int n, pad;
};

// ---- the fused gate step ------------------------------------------------------------------------
// The mixed finish: the same sweeps in double-float (FP32 pairs, on the FP32 pipes) on B (Bh, Bl: rows x k,
// ld rows) accumulating V (Vh, Vl: k x k, ld k).  Every lane forms the pair's compensated sums over its rows,
// the warp reduces them, and every lane derives the same rotation from the broadcast sums.
__device__ bool team_sweeps_df(const Team& T, float2* Bh, float2* Bl, float2* Vh, float2* Vl, int rows, int k, float tol,
                               float smax, int max_sweeps, float tan_stop, SweepCount cnt) {
  const int np = k + (k & 1), npairs = np / 2;
  bool converged = false;
  cnt.start(T);
  T.sync();
  for (int sweep = 0; sweep < max_sweeps && !converged; sweep++) {
    unsigned* sc = cnt.open(T, sweep);
    for (int round = 0; round < np - 1; round++) {
      for (int pair = T.warp; pair < npairs; pair += T.nw) {
        int p, q;
        round_pair(np, round, pair, p, q);
        if (q >= k) continue;
        const long cp = (long)rows * p, cq = (long)rows * q, dp = (long)k * p, dq = (long)k * q;
        float2 xh[TM_RPL], xl[TM_RPL], yh[TM_RPL], yl[TM_RPL], uh[TM_RPL], ul[TM_RPL], wh[TM_RPL], wl[TM_RPL];
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          const int r = T.lane + 32 * j;
          xh[j] = xl[j] = yh[j] = yl[j] = uh[j] = ul[j] = wh[j] = wl[j] = make_float2(0.f, 0.f);
          if (r < rows) {
            xh[j] = __ldcg(Bh + cp + r); xl[j] = __ldcg(Bl + cp + r);
            yh[j] = __ldcg(Bh + cq + r); yl[j] = __ldcg(Bl + cq + r);
          }
          if (r < k) {
            uh[j] = __ldcg(Vh + dp + r); ul[j] = __ldcg(Vl + dp + r);
            wh[j] = __ldcg(Vh + dq + r); wl[j] = __ldcg(Vl + dq + r);
          }
        }
        DotAcc a{0.f, 0.f}, b{0.f, 0.f}, gr{0.f, 0.f}, gi{0.f, 0.f};
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          if (32 * j >= rows) break;
          df_dot_acc(xh[j], xl[j], yh[j], yl[j], a, b, gr, gi);
        }
        const dfl k4 = df_warp_sum4_t(dot_final(a), dot_final(b), dot_final(gr), dot_final(gi));
        DfParams P;
        if (!rotation_params_df(df_shfl(k4, 0), df_shfl(k4, 8), df_shfl(k4, 16), df_shfl(k4, 24), tol, smax, P))
          continue;
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          const int r = T.lane + 32 * j;
          if (r < rows) {
            df_rot_any(xh[j], xl[j], yh[j], yl[j], P);
            __stcg(Bh + cp + r, xh[j]); __stcg(Bl + cp + r, xl[j]);
            __stcg(Bh + cq + r, yh[j]); __stcg(Bl + cq + r, yl[j]);
          }
          if (r < k) {
            df_rot_any(uh[j], ul[j], wh[j], wl[j], P);
            __stcg(Vh + dp + r, uh[j]); __stcg(Vl + dp + r, ul[j]);
            __stcg(Vh + dq + r, wh[j]); __stcg(Vl + dq + r, wl[j]);
          }
        }
        if (T.lane == 0) SweepCount::add(sc, P.tabs);
      }
      T.sync();
    }
    converged = SweepCount::done(sc, tan_stop);
  }
  T.sync();  // the counters have been read
  return converged;
}

// R = I - X^H X from X's transpose Xt (k x k, ld k), half of it computed: lanes on consecutive columns of X,
// column i with column i - d.  FP32 values of compensated double-float sums.
__device__ void team_gram_df(const Team& T, const float2* Th, const float2* Tl, int k, float2* R) {
  for (int t = T.tid; t < k * (k / 2 + 1); t += T.nt) {
    const int i = t % k, d = t / k, j = i >= d ? i - d : i - d + k;
    if (2 * d == k && i < j) continue;  // the pair's other end has it
    DotAcc re{0.f, 0.f}, im{0.f, 0.f};
    for (int x = 0; x < k; x++) {
      const float2 ah = Th[i + k * x], al = Tl[i + k * x], bh = Th[j + k * x], bl = Tl[j + k * x];
      dot2_step(re, ah.x, al.x, bh.x, bl.x);  // conj(a) b
      dot2_step(re, ah.y, al.y, bh.y, bl.y);
      dot2_step(im, ah.x, al.x, bh.y, bl.y);
      dot2_step(im, -ah.y, -al.y, bh.x, bl.x);
    }
    const dfl r = df_add({d == 0 ? 1.f : 0.f, 0.f}, df_neg(dot_final(re))), m = df_neg(dot_final(im));
    const float2 v = make_float2(r.h + r.l, d == 0 ? 0.f : m.h + m.l);
    R[i + k * j] = v;
    if (d) R[j + k * i] = make_float2(v.x, -v.y);
  }
}
// the same with FP64 sums of FP64 values
__device__ void team_gram(const Team& T, const double2* Xt, int k, float2* R) {
  for (int t = T.tid; t < k * (k / 2 + 1); t += T.nt) {
    const int i = t % k, d = t / k, j = i >= d ? i - d : i - d + k;
    if (2 * d == k && i < j) continue;  // the pair's other end has it
    double re = d == 0 ? -1.0 : 0.0, im = 0.0;
#pragma unroll 4
    for (int x = 0; x < k; x++) {
      const double2 a = Xt[i + k * x], b = Xt[j + k * x];
      re = fma(a.x, b.x, fma(a.y, b.y, re));
      im = fma(a.x, b.y, fma(-a.y, b.x, im));
    }
    const float2 v = make_float2((float)-re, d == 0 ? 0.f : (float)-im);
    R[i + k * j] = v;
    if (d) R[j + k * i] = make_float2(v.x, -v.y);
  }
}

// X_hi R / 2 at element t: FP32 products (|R| << 1)
__device__ __forceinline__ float2 half_product(const float2* Xh, const float2* R, int k, int t) {
  const int i = t % k, j = t / k;
  float ar = 0.f, ai = 0.f;
  for (int x = 0; x < k; x++) {
    const float2 a = Xh[i + (long)k * x], r = R[x + (long)k * j];
    ar = fmaf(a.x, r.x, fmaf(-a.y, r.y, ar));
    ai = fmaf(a.x, r.y, fmaf(a.y, r.x, ai));
  }
  return make_float2(0.5f * ar, 0.5f * ai);
}

// Y = X + X_hi R / 2 in double-float and its transpose; k x k, ld k.
__device__ void team_ns_df(const Team& T, const float2* Xh, const float2* Xl, const float2* R, int k, float2* Yh, float2* Yl,
                           float2* Th, float2* Tl) {
  for (int t = T.tid; t < k * k; t += T.nt) {
    const float2 a = half_product(Xh, R, k, t);
    const dfl yr = df_add_f({Xh[t].x, Xl[t].x}, a.x), yi = df_add_f({Xh[t].y, Xl[t].y}, a.y);
    Yh[t] = make_float2(yr.h, yi.h);
    Yl[t] = make_float2(yr.l, yi.l);
    if (Th) {
      const int tt = t / k + k * (t % k);
      Th[tt] = Yh[t];
      Tl[tt] = Yl[t];
    }
  }
}

// C = A X in double-float: A (Ah, Al) rows x k (ld rows), X (Xh, Xl) k x k, C rows x k (ld rows).
__device__ void team_gemm_df(const Team& T, const float2* Ah, const float2* Al, int rows, const float2* Xh,
                             const float2* Xl, int k, float2* Ch, float2* Cl) {
  for (int t = T.tid; t < rows * k; t += T.nt) {
    const int i = t % rows, j = t / rows;
    DotAcc re{0.f, 0.f}, im{0.f, 0.f};
    for (int x = 0; x < k; x++) {
      const float2 ah = Ah[i + (long)rows * x], al = Al[i + (long)rows * x];
      const float2 bh = Xh[x + (long)k * j], bl = Xl[x + (long)k * j];
      dot2_step(re, ah.x, al.x, bh.x, bl.x);
      dot2_step(re, -ah.y, -al.y, bh.y, bl.y);
      dot2_step(im, ah.x, al.x, bh.y, bl.y);
      dot2_step(im, ah.y, al.y, bh.x, bl.x);
    }
    const dfl r = dot_final(re), m = dot_final(im);
    Ch[t] = make_float2(r.h, m.h);
    Cl[t] = make_float2(r.l, m.l);
  }
}
__device__ void team_gemm(const Team& T, const double2* A, int rows, const double2* X, int k, double2* C) {
  for (int t = T.tid; t < rows * k; t += T.nt) {
    const int i = t % rows, j = t / rows;
    double2 c = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int x = 0; x < k; x++) {
      const double2 a = A[i + (long)rows * x], b = X[x + (long)k * j];
      c.x = fma(a.x, b.x, fma(-a.y, b.y, c.x));
      c.y = fma(a.x, b.y, fma(a.y, b.x, c.y));
    }
    C[t] = c;
  }
}

// W's first `keep` columns (rows x keep, ld rows, nearly unit) made orthonormal, each column's direction and
// phase kept: classical Gram-Schmidt twice.  A column's updates are dealt out by row, 8 lanes to a row.
__device__ void team_orthonormalise(const Team& T, double2* W, int rows, int keep, double2* coef) {
  for (int j = 0; j < keep; j++) {
    double2* wj = W + (long)rows * j;
    for (int pass = 0; pass < 2 && j > 0; pass++) {
      for (int i = T.warp; i < j; i += T.nw) {
        const double2* wi = W + (long)rows * i;
        double re = 0.0, im = 0.0;
        for (int r = T.lane; r < rows; r += 32) {
          const double2 x = wi[r], y = wj[r];
          re += x.x * y.x + x.y * y.y;
          im += x.x * y.y - x.y * y.x;
        }
        re = warp_sum(re);
        im = warp_sum(im);
        if (T.lane == 0) coef[i] = make_double2(re, im);
      }
      T.sync();
      for (int r0 = 4 * T.warp; r0 < rows; r0 += 4 * T.nw) {
        const int r = r0 + (T.lane >> 3);
        double2 v = make_double2(0.0, 0.0);
        if (r < rows)
          for (int i = T.lane & 7; i < j; i += 8) v = cadd(v, cmul(W[r + (long)rows * i], coef[i]));
        for (int o = 4; o > 0; o >>= 1) {
          v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
          v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (r < rows && (T.lane & 7) == 0) wj[r] = csub(wj[r], v);
      }
      T.sync();
    }
    if (j == 0) continue;
    // every warp forms the norm of the column, then scales its share of the rows
    double s = 0.0;
    for (int r = T.lane; r < rows; r += 32) s += wj[r].x * wj[r].x + wj[r].y * wj[r].y;
    s = warp_sum(s);
    const double inv = s > 0.0 ? 1.0 / sqrt(s) : 0.0;
    T.sync();
    for (int r = T.tid; r < rows; r += T.nt) wj[r] = cscale(wj[r], inv);
    T.sync();
  }
}

// One cluster per task (strided over the layer's tasks).  ws: slot_size(side) double2 per cluster.  dry = 1 runs
// the arithmetic without writing the chain (the autotuner's timing runs).
//
// The SVD: FP64 sweeps up to BT_PRE_MIN columns, team_svd (FP32 sweeps refined by FP64 products) up to
// BT_TEAM_MAX.  Above that FP32 sweeps on a copy of theta (64x the FP64 rate on this part), two Newton-Schulz
// steps X <- X + X (I - X^H X) / 2 that make their rotations unitary to rounding, B = theta X, and full-precision
// sweeps that finish from couplings of ~1e-6 in two or three: in FP64, or with MIXED in double-float on the FP32 pipes.
//
// What bounds a step is its chain of rounds: 127 of them in a sweep of 128 columns.  On one CTA a
// double-float sweep of theta 128 x 128 needs 1.4 ms of its SM's FP32 rate and an FP64 sweep ~10, so a layer of
// saturated bonds took 20 ms while most SMs idled.  A cluster deals the rounds' pairs out to up to 8 SMs, and
// the FP32 sweeps run 15 rounds a sweep on Gram matrices.
template <bool MIXED>
__global__ void __launch_bounds__(512, 1)
    batch_gate_k(const BTask* __restrict__ tasks, int ntasks, double2* __restrict__ ws, int side, int dry, int team) {
  __shared__ BTask T;
  __shared__ double2 G[16];
  __shared__ double sig[BT_MAXK], srt[BT_MAXK];
  __shared__ int perm[BT_MAXK];
  __shared__ double scale_f, smax_s;
  __shared__ int keep_s, reorth_s;
  __shared__ GrShared<TM_W> gsh;
  __shared__ __align__(16) float2 tile[TM_TILE];
  Team M;
  M.size = team;
  M.rank = blockIdx.x % team;
  M.tid = M.rank * blockDim.x + threadIdx.x;
  M.nt = team * blockDim.x;
  M.lane = threadIdx.x & 31;
  M.warp = M.tid >> 5;
  M.nw = M.nt >> 5;
  const int tid = threadIdx.x;
  const size_t K2 = (size_t)side * side;
  double2* TH = ws + (size_t)(blockIdx.x / team) * (4 * K2 + TM_SQUARES * K2 + TM_MAXK + 2 * BT_MAXK);
  double2 *B = TH + K2, *V = B + K2, *W = V + K2, *coef = W + K2, *S0 = coef + 2 * BT_MAXK, *S1 = S0 + K2, *S2 = S1 + K2;
  double* nrm = reinterpret_cast<double*>(coef + BT_MAXK);
  const SweepCount cnt{reinterpret_cast<unsigned*>(nrm + BT_MAXK)};

  for (int ti = blockIdx.x / team; ti < ntasks; ti += gridDim.x / team) {
    if (tid == 0) T = tasks[ti];
    __syncthreads();
    if (tid < 16) G[tid] = T.gate[tid];
    const int b = T.bond;
    const int cl = b > 0 ? T.bd[b - 1] : 1, cc = T.bd[b], cr = b + 1 < T.nb ? T.bd[b + 1] : 1;
    const int m = 2 * cl, nn = 2 * cr;
    const bool tall = m >= nn;
    const int rows = tall ? m : nn, k = tall ? nn : m;
    const bool lam_on = T.haslam[b] != 0;
    const bool sweep = k <= BT_PRE_MIN, wide = k > BT_TEAM_MAX;
    __syncthreads();

    // ---- theta' = G (A_l diag(Lambda) A_r), into TH (tall) or TH = theta'^H (wide)
    for (int t = M.tid; t < cl * cr; t += M.nt) {
      const int l = t % cl, r = t / cl;
      double2 acc[2][2];
      acc[0][0] = acc[0][1] = acc[1][0] = acc[1][1] = make_double2(0.0, 0.0);
#pragma unroll 2
      for (int x = 0; x < cc; x++) {
        const double w = lam_on ? T.lam[x] : 1.0;
        const double2 a0 = cscale(T.sl[l + (long)cl * (2 * x)], w), a1 = cscale(T.sl[l + (long)cl * (1 + 2 * x)], w);
        const double2 b0 = T.sr[x + (long)cc * (2 * r)], b1 = T.sr[x + (long)cc * (1 + 2 * r)];
        cfma(acc[0][0], a0, b0);
        cfma(acc[0][1], a0, b1);
        cfma(acc[1][0], a1, b0);
        cfma(acc[1][1], a1, b1);
      }
#pragma unroll
      for (int p1 = 0; p1 < 2; p1++)
#pragma unroll
        for (int p2 = 0; p2 < 2; p2++) {
          double2 v = make_double2(0.0, 0.0);
#pragma unroll
          for (int o1 = 0; o1 < 2; o1++)
#pragma unroll
            for (int o2 = 0; o2 < 2; o2++) cfma(v, G[(2 * p1 + p2) * 4 + 2 * o1 + o2], acc[o1][o2]);
          const int rt = l + cl * p1, ct = p2 + 2 * r;
          if (tall) TH[rt + (long)rows * ct] = v;
          else TH[ct + (long)rows * rt] = cconj(v);
        }
    }
    M.sync();

    // ---- column norms, power-of-two prescale (sigma_max of the scaled columns in [1/2, 1))
    team_norms(M, TH, rows, k, nrm, sig);
    if (tid < 32) {
      double mx = 0.0;
      for (int j = tid; j < k; j += 32) mx = fmax(mx, sig[j]);
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (tid == 0) {
        int e = 0;
        if (mx > 0.0) frexp(mx, &e);
        scale_f = ldexp(1.0, e);
        smax_s = mx > 0.0 ? ldexp(mx, -e) : 0.0;
      }
    }
    __syncthreads();
    const double smax = smax_s;
    {
      // (copies for the FP32 sweeps: B32 | V32)
      const double inv = 1.0 / scale_f;
      float2* B32 = reinterpret_cast<float2*>(S0);
      for (int t = M.tid; t < rows * k; t += M.nt) {
        const double2 v = cscale(TH[t], inv);
        (sweep ? B : TH)[t] = v;
        if (wide) B32[t] = make_float2((float)v.x, (float)v.y);
      }
      for (int t = M.tid; t < k * k; t += M.nt) {
        const bool d = (t % k) == (t / k);
        if (wide) B32[K2 + t] = make_float2(d ? 1.f : 0.f, 0.f);
        if (sweep) V[t] = make_double2(d ? 1.0 : 0.0, 0.0);
      }
    }
    M.sync();

    // ---- B = theta V with orthogonal columns: FP64 sweeps, a refinement, or sweeps preconditioned in FP32
    const double tol = sqrt((double)rows) * Eps<double>::v;
    bool converged = false;
    if (sweep) {
      converged = team_sweeps(M, B, V, rows, k, tol, smax, BT_MAX_SWEEPS, 1e-8f, cnt);
    } else if (!wide) {
      converged = team_svd(M, TH, B, V, rows, k, tol, smax, S0, side, gsh, tile);
    } else {
      float2 *B32 = reinterpret_cast<float2*>(S0), *V32 = B32 + K2;
      const float tol32 = fmaxf(4e-6f, 2.f * sqrtf((float)rows) * Eps<float>::v);
      team_sweeps_f32(M, B32, V32, rows, k, tol32, (float)smax, 20, 0.15f, cnt, gsh, tile);
      if (MIXED) {
        // halves of the squares: S0 B32 | X0 -> B' (hi | lo), S1 theta (hi | lo), S2 X0's transpose -> X1's
        // (hi | lo) -> X2 (hi | lo), W X1 (hi | lo), V R | zeros
        float2 *h0 = reinterpret_cast<float2*>(S0), *h1 = reinterpret_cast<float2*>(S1), *h2 = reinterpret_cast<float2*>(S2);
        float2 *hV = reinterpret_cast<float2*>(V), *hW = reinterpret_cast<float2*>(W);
        float2 *X0 = V32, *zero = hV + K2;
        for (int t = M.tid; t < k * k; t += M.nt) {
          h2[t / k + k * (t % k)] = X0[t];
          zero[t] = make_float2(0.f, 0.f);
        }
        for (int t = M.tid; t < rows * k; t += M.nt) {
          const dfl re = df_from(TH[t].x), im = df_from(TH[t].y);
          h1[t] = make_float2(re.h, im.h);
          h1[K2 + t] = make_float2(re.l, im.l);
        }
        M.sync();
        team_gram_df(M, h2, zero, k, hV);  // 1e-6 -> 1e-12 -> rounding
        M.sync();
        team_ns_df(M, X0, zero, hV, k, hW, hW + K2, h2, h2 + K2);
        M.sync();
        team_gram_df(M, h2, h2 + K2, k, hV);
        M.sync();
        float2 *Xh = h2, *Xl = h2 + K2;  // (the transposes have been read)
        team_ns_df(M, hW, hW + K2, hV, k, Xh, Xl, nullptr, nullptr);
        M.sync();
        team_gemm_df(M, h1, h1 + K2, rows, Xh, Xl, k, h0, h0 + K2);
        const float toldf = (float)(32.0 * sqrt((double)rows) * Eps<double>::v);
        converged = team_sweeps_df(M, h0, h0 + K2, Xh, Xl, rows, k, toldf, (float)smax, BT_MAX_SWEEPS, 1e-7f, cnt);
        for (int t = M.tid; t < rows * k; t += M.nt) {
          const float2 h = h0[t], l = h0[K2 + t];
          B[t] = make_double2((double)h.x + l.x, (double)h.y + l.y);
        }
        for (int t = M.tid; t < k * k; t += M.nt) {
          const float2 h = Xh[t], l = Xl[t];
          V[t] = make_double2((double)h.x + l.x, (double)h.y + l.y);
        }
        M.sync();
      } else {
        // the same in FP64 (the steps' corrections X R / 2 in FP32, |R| ~ 1e-6 and 1e-12; the first step's
        // R needs no more than double-float sums): S1 X0's transpose | zeros -> X2, S2 X1's transpose, W X1,
        // V R | X1 hi
        double2 *Xt = S2, *X1 = W;
        float2 *R = reinterpret_cast<float2*>(V), *Xf = R + K2, *Tf = reinterpret_cast<float2*>(S1);
        for (int t = M.tid; t < k * k; t += M.nt) {
          Tf[t / k + k * (t % k)] = V32[t];
          Tf[K2 + t] = make_float2(0.f, 0.f);
        }
        M.sync();
        team_gram_df(M, Tf, Tf + K2, k, R);
        M.sync();
        for (int t = M.tid; t < k * k; t += M.nt) {
          const float2 a = half_product(V32, R, k, t);
          const double2 v = make_double2((double)V32[t].x + a.x, (double)V32[t].y + a.y);
          X1[t] = v;
          Xt[t / k + k * (t % k)] = v;
          Xf[t] = make_float2((float)v.x, (float)v.y);
        }
        M.sync();
        team_gram(M, Xt, k, R);
        M.sync();
        for (int t = M.tid; t < k * k; t += M.nt) {
          const float2 a = half_product(Xf, R, k, t);
          S1[t] = make_double2(X1[t].x + a.x, X1[t].y + a.y);
        }
        M.sync();
        team_gemm(M, TH, rows, S1, k, S0);
        M.sync();
        for (int t = M.tid; t < rows * k; t += M.nt) B[t] = S0[t];
        for (int t = M.tid; t < k * k; t += M.nt) V[t] = S1[t];
        converged = team_sweeps(M, B, V, rows, k, tol, smax, BT_MAX_SWEEPS, 1e-8f, cnt);
      }
    }
    if (!converged && M.tid == 0) atomicExch(T.status, (int)QR_ENOCONV);

    // ---- sigma, descending order (ranks_before), truncation on the device
    team_norms(M, B, rows, k, nrm, sig);
    for (int j = tid; j < k; j += blockDim.x) {
      int rank = 0;
      const double v = sig[j];
      for (int i = 0; i < k; i++) rank += ranks_before(sig[i], i, v, j);
      perm[rank] = j;
      srt[rank] = v;
    }
    __syncthreads();
    if (tid == 0) {
      const int upto = T.maxdim >= 0 && T.maxdim < k ? T.maxdim : k;
      const double thr = isnan(T.threshold) ? 1e-16 : T.threshold;
      int kp = 0;
      while (kp < upto && fabs(srt[kp] * scale_f) > thr) kp++;
      if (kp == 0) {  // the chain would be left with an empty bond: keep one vector, flag the request
        if (M.rank == 0) atomicExch(T.status, (int)QR_EINVAL);
        kp = 1;
      }
      keep_s = kp;
      reorth_s = !(srt[kp - 1] > 1e-3 * srt[0]);
    }
    __syncthreads();
    const int keep = keep_s;

    // ---- the kept left vectors of B (columns perm[j] / sigma) into W
    for (int t = M.tid; t < rows * keep; t += M.nt) {
      const int r = t % rows, j = t / rows;
      const double s = srt[j];
      W[r + (long)rows * j] = s > 0.0 ? cscale(B[r + (long)rows * perm[j]], 1.0 / s) : make_double2(0.0, 0.0);
    }
    M.sync();
    if (reorth_s) team_orthonormalise(M, W, rows, keep, coef);

    // ---- write-back: A_l (cl, 2, keep), A_r (keep, 2, cr), Lambda, bond dimension
    if (!dry) {
      if (tall) {  // theta = W S (V[:, perm])^H
        for (int t = M.tid; t < m * keep; t += M.nt) T.sl[t] = W[t % m + (long)rows * (t / m)];
        for (int t = M.tid; t < keep * nn; t += M.nt) {
          const int j = t % keep, col = t / keep;
          T.sr[t] = cconj(V[col + (long)k * perm[j]]);
        }
      } else {  // theta^H = W S V^H  =>  theta = V[:, perm] S W^H
        for (int t = M.tid; t < m * keep; t += M.nt) {
          const int row = t % m, j = t / m;
          T.sl[t] = V[row + (long)k * perm[j]];
        }
        for (int t = M.tid; t < keep * nn; t += M.nt) {
          const int j = t % keep, col = t / keep;
          T.sr[t] = cconj(W[col + (long)rows * j]);
        }
      }
      for (int j = M.tid; j < keep; j += M.nt) T.lam[j] = srt[j] * scale_f;
      if (M.tid == 0) {
        T.bd[b] = keep;
        T.haslam[b] = 1;
      }
    }
    M.sync();
  }
}

// ---- expectation values of Pauli strings: one cluster per string, FP64 environment sweep --------
// E[a, a'] (ket a, bra a') from the left; per site X[a', o, r] = sum_a E[a, a'] A[a, o, r], then
// E'[r, r'] = sum_{a', o'} conj(A[a', o', r']) sum_o P[o', o] X[a', o, r], times Lambda_r Lambda_r'
// when the bond to the right holds a Lambda.  A Pauli string's environment is Hermitian, so half of
// E' is computed and E[a, a'] is read as conj(E[a', a]), which puts the lanes on consecutive values.
//
// Bound by the FP64 rate of the SMs that work on the longest chain: 6 chi^3 complex multiply-adds a
// site at 0.5 DFMA per clock and scheduler.  So the columns r of a site are dealt to the CTAs of a
// cluster: X for a CTA's own columns stays in its shared memory, E goes through L2, and one cluster
// barrier ends the site.  The longest of 64 strings (40 sites, chi 64) took 47.7 ms on one CTA.
// ws: 2 * 64 * 64 double2 per string.
constexpr int BX_CL = 8;     // CTAs per string
constexpr int BX_NT = 384;   // 9 warps' worth of E' at chi = 64: three per scheduler at most
constexpr int BX_OWN = (BT_MAXCHI + BX_CL - 1) / BX_CL;

// the part of pauli code's row op in (P x)[op] for x = (x0, x1)
__device__ __forceinline__ double2 pauli_apply(int code, int op, const double2& x0, const double2& x1) {
  switch (code) {
    case 1: return op == 0 ? x1 : x0;                                                    // X
    case 2: return op == 0 ? make_double2(x1.y, -x1.x) : make_double2(-x0.y, x0.x);      // Y
    case 3: return op == 0 ? x0 : make_double2(-x1.x, -x1.y);                            // Z
    default: return op == 0 ? x0 : x1;                                                   // I
  }
}

__global__ void __launch_bounds__(BX_NT) batch_expect_k(const BObs* __restrict__ obs, double2* __restrict__ ws) {
  __shared__ double2 X[(2 * BT_MAXCHI + 1) * BX_OWN];
  const int str = blockIdx.x / BX_CL, rank = blockIdx.x % BX_CL;
  const BObs O = obs[str];
  double2* E0 = ws + (size_t)str * 2 * BT_MAXCHI * BT_MAXCHI;
  double2* E1 = E0 + BT_MAXCHI * BT_MAXCHI;
  if (rank == 0 && threadIdx.x == 0) E0[0] = make_double2(1.0, 0.0);
  __syncwarp();
  cluster_sync_all();
  for (int i = 0; i < O.n; i++) {
    const double2* A = O.sites[i];
    const int cl = i > 0 ? O.bd[i - 1] : 1, cr = i + 1 < O.n ? O.bd[i] : 1;
    const int code = O.pauli[i];
    const int r0 = cr * rank / BX_CL, own = cr * (rank + 1) / BX_CL - r0, ld = 2 * cl + 1;
    // X[a', o, r] (a' fastest) of the own columns
    for (int t = threadIdx.x; t < cl * 2 * own; t += BX_NT) {
      const int ap = t % cl, orr = t / cl;  // orr = o + 2 (r - r0)
      const double2* col = A + (long)cl * (2 * r0 + orr);
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
      for (int a = 0; a < cl; a++) {
        const double2 e = __ldcg(E0 + ap + cl * a), v = col[a];
        acc.x = fma(e.x, v.x, fma(e.y, v.y, acc.x));
        acc.y = fma(e.x, v.y, fma(-e.y, v.x, acc.y));
      }
      X[(orr >> 1) * ld + (orr & 1) * cl + ap] = acc;
    }
    __syncthreads();
    const bool lam_on = i + 1 < O.n && O.haslam[i];
    const double* lam = lam_on ? O.lams[i] : nullptr;
    // row r of E' meets r' = r, r + 1, .. r + cr / 2 (mod cr): every CTA has the same share of the pairs
    const int half = cr / 2 + 1;
    for (int t = threadIdx.x; t < own * half; t += BX_NT) {
      const int rl = t % own, j = t / own, r = r0 + rl;
      int rp = r + j;
      if (rp >= cr) rp -= cr;
      if (2 * j == cr && rp < r) continue;  // the other end of this pair has it
      const double2* x = X + rl * ld;
      const double2* col = A + (long)cl * 2 * rp;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 2
      for (int ap = 0; ap < cl; ap++) {
        const double2 x0 = x[ap], x1 = x[cl + ap];
#pragma unroll
        for (int op = 0; op < 2; op++) {
          const double2 y = pauli_apply(code, op, x0, x1), v = col[ap + cl * op];
          acc.x = fma(v.x, y.x, fma(v.y, y.y, acc.x));
          acc.y = fma(v.x, y.y, fma(-v.y, y.x, acc.y));
        }
      }
      if (lam_on) acc = cscale(acc, lam[r] * lam[rp]);
      if (j == 0) acc.y = 0.0;
      __stcg(E1 + r + cr * rp, acc);
      if (j) __stcg(E1 + rp + cr * r, cconj(acc));
    }
    __syncwarp();
    cluster_sync_all();
    double2* tmp = E0;
    E0 = E1;
    E1 = tmp;
  }
  if (rank == 0 && threadIdx.x == 0) O.out[0] = __ldcg(E0);
}

// state init: every site of every chain becomes |0> = (1, 0) in a (1, 2, 1) array
__global__ void batch_init_k(double2* const* __restrict__ sites, int nsites) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nsites; t += gridDim.x * blockDim.x) {
    sites[t][0] = make_double2(1.0, 0.0);
    sites[t][1] = make_double2(0.0, 0.0);
  }
}

// synthetic sites for the autotuner: deterministic values of unit magnitude scale
__global__ void batch_fill_k(double2* p, long count, double scale) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < count; t += (long)gridDim.x * blockDim.x) {
    const unsigned h1 = (unsigned)(t * 2654435761u) ^ 0x9e3779b9u, h2 = (unsigned)(t * 40503u + 12345u) * 2246822519u;
    p[t] = make_double2(scale * ((double)(h1 & 0xffffff) / 16777216.0 - 0.5),
                        scale * ((double)(h2 & 0xffffff) / 16777216.0 - 0.5));
  }
}

// clusters x cl CTAs of nt threads
template <typename... P, typename... A>
cudaError_t launch_cluster(void (*kern)(P...), unsigned clusters, int cl, int nt, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * cl);
  cfg.blockDim = dim3(nt);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

int cap_of(int n, int b, int chi_max) {
  const int e = std::min(b + 1, n - b - 1);
  long c = e >= 30 ? (1L << 30) : (1L << e);
  return (int)std::min<long>(c, chi_max);
}

struct BReq {
  int n = 0, chi_max = 0;
  double threshold = 1e-10;
  std::vector<int> gsite;
  std::vector<double2> gmat;  // 16 per gate
  std::vector<int> ow, os, op;
  // results
  int status = QR_OK;
  std::vector<double2> values;
  std::vector<int> bd;
  std::vector<std::vector<double>> lam;
  std::vector<int> layer_of_gate;
};

// CTAs per gate step of theta up to k x k: as many as have work in a round.  A round of the sweeps has
// k / 2 pairs (a warp each, at least 4 warps a CTA) and one of the FP32 sweeps k / 16 items.
int team_size(int k) { return k > 64 ? BT_MAXTEAM : k > 16 ? 4 : 1; }

// Autotuner cache: (device name, chi class) -> warps per CTA of the layer kernel
std::mutex g_tune_mu;
std::map<std::string, int> g_tune;

// The launch of a layer: the largest theta that its bonds can have reached, CTAs per gate step and clusters.  Four
// CTAs of 128 threads a SM fill the GPU; more clusters would only want more workspace.
struct Layer {
  int side = 2, team = 1, clusters = 1;
  size_t ws() const { return slot_size(side) * clusters; }
};
void size_layer(Layer& l, int ntasks, int sms) {
  l.team = team_size(l.side);
  l.clusters = std::max(1, std::min(ntasks, 4 * sms / l.team));
}
std::vector<Layer> plan_layers(const std::vector<BReq>& reqs, int nlayers, int sms) {
  std::vector<Layer> out(nlayers);
  std::vector<int> ntasks(nlayers, 0);
  for (const BReq& r : reqs) {
    std::vector<int> ub(r.n - 1, 1);  // bounds of the bond dimensions after the gates so far
    for (size_t g = 0; g < r.gsite.size(); g++) {
      const int b = r.gsite[g], m = 2 * (b > 0 ? ub[b - 1] : 1), n = 2 * (b + 1 < r.n - 1 ? ub[b + 1] : 1);
      Layer& l = out[r.layer_of_gate[g]];
      l.side = std::max(l.side, std::max(m, n));
      ntasks[r.layer_of_gate[g]]++;
      ub[b] = std::min(std::min(m, n), cap_of(r.n, b, r.chi_max));
    }
  }
  for (int L = 0; L < nlayers; L++) size_layer(out[L], ntasks[L], sms);
  return out;
}

std::string tune_file() {
  const char* p = getenv("QROCHET_TUNE_FILE");
  return p ? std::string(p) : std::string();
}

void tune_load() {
  static bool loaded = false;
  if (loaded) return;
  loaded = true;
  const std::string f = tune_file();
  if (f.empty()) return;
  FILE* fp = fopen(f.c_str(), "r");
  if (!fp) return;
  char key[256];
  int v = 0;
  // keep only choices the autotuner can make itself (4, 8 or 16 warps): the layer kernel's
  // shape depends on it, so a damaged or hand-edited entry is re-tuned instead of launched
  while (fscanf(fp, "%255s %d", key, &v) == 2)
    if (v == 4 || v == 8 || v == 16) g_tune[key] = v;
  fclose(fp);
}

void tune_save() {
  const std::string f = tune_file();
  if (f.empty()) return;
  FILE* fp = fopen(f.c_str(), "w");
  if (!fp) return;
  for (auto& kv : g_tune) fprintf(fp, "%s %d\n", kv.first.c_str(), kv.second);
  fclose(fp);
}

}  // namespace
}  // namespace qr

using namespace qr;

struct qr_batch {
  int device = 0;
  int precision = QR_FP64;
  std::vector<BReq> reqs;
  bool ran = false;
  int warps = 0, layers = 0, launches = 0, tuned_from_cache = 0;
  size_t graph_nodes = 0;
  double run_ms = 0.0, tune_ms = 0.0;
  std::vector<double> tune_candidates_ms;
};

namespace {
// the tuning cache's key of the batch's largest bond class, and the choice that it holds (0: none yet)
int tune_key(const qr_batch* bt, int chi, std::string* out) {
  cudaDeviceProp prop;
  QR_CUDA(cudaGetDeviceProperties(&prop, bt->device));
  const bool mixed = (bt->precision & QR_MIXED) != 0;
  std::string key = std::string(prop.name).substr(0, 40) + "/chi" + std::to_string(chi) + (mixed ? "/mixed" : "/fp64");
  for (char& ch : key)
    if (ch == ' ') ch = '_';
  *out = key;
  return QR_OK;
}
int tuned_warps(const std::string& key) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  tune_load();
  auto it = g_tune.find(key);
  return it != g_tune.end() ? it->second : 0;
}

// warps per CTA for the layer kernel at bond class `chi` (the batch's largest), measured on
// synthetic gate steps of that class in dry mode (no chain is written)
int autotune(qr_batch* bt, cudaStream_t s, const std::string& key, int chi, const Layer& l, double2* ws) {
  const bool mixed = (bt->precision & QR_MIXED) != 0;
  // synthetic chain of 3 bonds at chi on both sides of the middle one
  const int ntask = l.clusters;
  const size_t site = (size_t)chi * 2 * chi;
  double2* sites = nullptr;
  double* lam = nullptr;
  int* ints = nullptr;
  BTask* dt = nullptr;
  QR_CUDA(cudaMallocAsync((void**)&sites, sizeof(double2) * (2 * site + 16), s));
  QR_CUDA(cudaMallocAsync((void**)&lam, sizeof(double) * chi, s));
  QR_CUDA(cudaMallocAsync((void**)&ints, sizeof(int) * 8, s));
  QR_CUDA(cudaMallocAsync((void**)&dt, sizeof(BTask) * ntask, s));
  batch_fill_k<<<256, 256, 0, s>>>(sites, (long)(2 * site + 16), 1.0 / chi);
  count_launch();
  int hi[8] = {chi, chi, chi, 0, 0, 0, 0, 0};
  QR_CUDA(cudaMemcpyAsync(ints, hi, sizeof(hi), cudaMemcpyHostToDevice, s));
  std::vector<BTask> ht(ntask);
  for (int i = 0; i < ntask; i++) {
    BTask& t = ht[i];
    t.sl = sites;
    t.sr = sites + site;
    t.lam = lam;
    t.bd = ints;
    t.haslam = ints + 3;
    t.gate = sites + 2 * site;
    t.status = reinterpret_cast<int*>(ints + 7);
    t.threshold = 1e-10;
    t.bond = 1;
    t.nb = 3;
    t.maxdim = chi;
  }
  QR_CUDA(cudaMemcpyAsync(dt, ht.data(), sizeof(BTask) * ntask, cudaMemcpyHostToDevice, s));
  cudaEvent_t e0, e1;
  QR_CUDA(cudaEventCreate(&e0));
  QR_CUDA(cudaEventCreate(&e1));
  const int cand[3] = {4, 8, 16};
  float best = 1e30f;
  int bw = 8;
  bt->tune_candidates_ms.clear();
  for (int w : cand) {
    auto kern = mixed ? batch_gate_k<true> : batch_gate_k<false>;
    QR_CUDA(launch_cluster(kern, ntask, l.team, 32 * w, s, dt, ntask, ws, l.side, 1, l.team));  // warm-up
    count_launch();
    QR_CUDA(cudaEventRecord(e0, s));
    QR_CUDA(launch_cluster(kern, ntask, l.team, 32 * w, s, dt, ntask, ws, l.side, 1, l.team));
    count_launch();
    QR_CUDA(cudaEventRecord(e1, s));
    QR_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    QR_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    bt->tune_candidates_ms.push_back(ms);
    bt->tune_ms += ms;
    if (ms < best) { best = ms; bw = w; }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(sites, s);
  cudaFreeAsync(lam, s);
  cudaFreeAsync(ints, s);
  cudaFreeAsync(dt, s);
  QR_CUDA(cudaGetLastError());
  bt->warps = bw;
  std::lock_guard<std::mutex> lk(g_tune_mu);
  g_tune[key] = bw;
  tune_save();
  return QR_OK;
}
}  // namespace

extern "C" {

int qr_batch_create(int device, qr_batch** out) try {
  if (!out) return fail(QR_EINVAL, "null output");
  qr_batch* b = new qr_batch();
  b->device = device;
  *out = b;
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_set_precision(qr_batch* b, int mode) try {
  if (!b) return fail(QR_EINVAL, "null batch");
  if (b->ran) return fail(QR_EINVAL, "the batch has already run");
  if (mode < 0 || mode > 3) return fail(QR_EINVAL, "bad precision");
  b->precision = mode;
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_free(qr_batch* b) try {
  delete b;
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_add(qr_batch* bt, int n, int chi_max, double threshold, int ngates, const int* gate_site,
                 const double* gate_mats, int nobs, const int* obs_weight, const int* obs_sites, const int* obs_paulis,
                 int* id) try {
  if (!bt || !id) return fail(QR_EINVAL, "null argument");
  if (bt->ran) return fail(QR_EINVAL, "the batch has already run");
  if (n < 2 || chi_max < 1) return fail(QR_EINVAL, "a request needs n >= 2 sites and chi_max >= 1");
  if (chi_max > BT_MAXCHI)
    return fail(QR_EINVAL, "the batched engine takes chi_max <= 64 (theta up to 128 x 128); serve larger requests");
  if (ngates < 0 || (ngates > 0 && (!gate_site || !gate_mats))) return fail(QR_EINVAL, "bad gate list");
  if (nobs < 0 || (nobs > 0 && (!obs_weight || !obs_sites || !obs_paulis))) return fail(QR_EINVAL, "bad observable list");
  BReq r;
  r.n = n;
  r.chi_max = chi_max;
  r.threshold = threshold;
  // layers: a gate opens a new layer when it shares a site with a gate of the current one
  std::vector<int> last_layer(n, -1);
  int cur = 0;
  std::vector<char> used(n, 0);
  for (int g = 0; g < ngates; g++) {
    const int s0 = gate_site[g];
    if (s0 < 0 || s0 + 1 >= n) return fail(QR_EINVAL, "gate site out of range");
    if (used[s0] || used[s0 + 1]) {
      cur++;
      std::fill(used.begin(), used.end(), 0);
    }
    used[s0] = used[s0 + 1] = 1;
    r.gsite.push_back(s0);
    r.layer_of_gate.push_back(cur);
    for (int e = 0; e < 16; e++) r.gmat.push_back(make_double2(gate_mats[32 * g + 2 * e], gate_mats[32 * g + 2 * e + 1]));
  }
  int pos = 0;
  for (int o = 0; o < nobs; o++) {
    if (obs_weight[o] < 0) return fail(QR_EINVAL, "bad observable weight");
    for (int w = 0; w < obs_weight[o]; w++, pos++) {
      if (obs_sites[pos] < 0 || obs_sites[pos] >= n || obs_paulis[pos] < 0 || obs_paulis[pos] > 3)
        return fail(QR_EINVAL, "bad Pauli string entry");
    }
    r.ow.push_back(obs_weight[o]);
  }
  r.os.assign(obs_sites, obs_sites + pos);
  r.op.assign(obs_paulis, obs_paulis + pos);
  bt->reqs.push_back(std::move(r));
  *id = (int)bt->reqs.size() - 1;
  return QR_OK;
} QR_ABI_CATCH

// layer index of every gate of request `id` (host-side schedule; no device needed)
int qr_batch_plan(const qr_batch* bt, int id, int* layer_of_gate, int* nlayers) try {
  if (!bt || id < 0 || id >= (int)bt->reqs.size()) return fail(QR_EINVAL, "bad batch request id");
  const BReq& r = bt->reqs[id];
  int mx = -1;
  for (size_t g = 0; g < r.layer_of_gate.size(); g++) {
    if (layer_of_gate) layer_of_gate[g] = r.layer_of_gate[g];
    mx = std::max(mx, r.layer_of_gate[g]);
  }
  if (nlayers) *nlayers = mx + 1;
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_run(qr_batch* bt, double* ms) try {
  if (!bt) return fail(QR_EINVAL, "null batch");
  if (bt->ran) return fail(QR_EINVAL, "the batch has already run");
  if (bt->reqs.empty()) return fail(QR_EINVAL, "empty batch");
  QR_CUDA(cudaSetDevice(bt->device));
  cudaStream_t s;
  QR_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sg{s};
  const int R = (int)bt->reqs.size();

  // ---- device layout: one allocation holding every buffer
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) / 256 * 256; return o; };
  struct ROff { size_t site0, lam0, bd, hl, sp, lp, gates, paulis, out, status; std::vector<size_t> site, lam; };
  std::vector<ROff> ro(R);
  int maxchi = 1, nlayers = 0, nobs_total = 0, nsites_total = 0;
  for (int q = 0; q < R; q++) {
    const BReq& r = bt->reqs[q];
    ROff& o = ro[q];
    o.site.resize(r.n);
    o.lam.resize(r.n - 1);
    for (int i = 0; i < r.n; i++) {
      const int cl = i > 0 ? cap_of(r.n, i - 1, r.chi_max) : 1, cr = i + 1 < r.n ? cap_of(r.n, i, r.chi_max) : 1;
      o.site[i] = take(sizeof(double2) * (size_t)cl * 2 * cr);
      maxchi = std::max(maxchi, std::max(cl, cr));
    }
    nsites_total += r.n;
    nobs_total += (int)r.ow.size();
    for (int L : r.layer_of_gate) nlayers = std::max(nlayers, L + 1);
  }
  // The tables are one block, [Lambda | values | bonds, flags, status | pointers, gates, strings, tasks]: the
  // start of its third part is uploaded with one copy, and its first three parts come back with one.  (A copy
  // per array took 9 ms of host time at 32 requests.)
  const size_t o_results = off;
  for (int q = 0; q < R; q++) {
    const BReq& r = bt->reqs[q];
    for (int b = 0; b < r.n - 1; b++) ro[q].lam[b] = take(sizeof(double) * cap_of(r.n, b, r.chi_max));
    ro[q].out = take(sizeof(double2) * std::max<size_t>(1, r.ow.size()));
  }
  const size_t o_image = off;
  for (int q = 0; q < R; q++) {
    const BReq& r = bt->reqs[q];
    ro[q].bd = take(sizeof(int) * (r.n - 1));
    ro[q].hl = take(sizeof(int) * (r.n - 1));
    ro[q].status = take(sizeof(int));
  }
  const size_t o_results_end = off;
  for (int q = 0; q < R; q++) {
    const BReq& r = bt->reqs[q];
    ro[q].sp = take(sizeof(double2*) * r.n);
    ro[q].lp = take(sizeof(double*) * (r.n - 1));
    ro[q].gates = take(sizeof(double2) * std::max<size_t>(1, r.gmat.size()));
    ro[q].paulis = take(sizeof(int) * (size_t)r.n * std::max<size_t>(1, r.ow.size()));
  }
  // per-layer task tables, larger bond classes first inside a layer
  std::vector<std::vector<std::pair<int, int>>> layer_tasks(nlayers);  // (request, gate)
  for (int q = 0; q < R; q++)
    for (size_t g = 0; g < bt->reqs[q].gsite.size(); g++) layer_tasks[bt->reqs[q].layer_of_gate[g]].push_back({q, (int)g});
  size_t ntask_total = 0;
  for (auto& L : layer_tasks) {
    std::stable_sort(L.begin(), L.end(), [&](const std::pair<int, int>& x, const std::pair<int, int>& y) {
      const BReq& a = bt->reqs[x.first];
      const BReq& c = bt->reqs[y.first];
      return cap_of(a.n, a.gsite[x.second], a.chi_max) > cap_of(c.n, c.gsite[y.second], c.chi_max);
    });
    ntask_total += L.size();
  }
  const size_t o_tasks = take(sizeof(BTask) * std::max<size_t>(1, ntask_total));
  const size_t o_obs = take(sizeof(BObs) * std::max(1, nobs_total));
  const size_t o_sites_tab = take(sizeof(double2*) * nsites_total);
  int sms = 0;
  QR_TRY(device_sm_count(&sms));
  const size_t o_image_end = off;
  const std::vector<Layer> layers = plan_layers(bt->reqs, nlayers, sms);
  const int tune_chi = std::min(maxchi, BT_MAXCHI);
  std::string key;
  QR_TRY(tune_key(bt, tune_chi, &key));
  bt->warps = tuned_warps(key);
  bt->tuned_from_cache = bt->warps != 0;
  Layer tune_layer;
  tune_layer.side = 2 * tune_chi;
  size_layer(tune_layer, 4 * sms, sms);
  size_t ws_words = bt->warps ? 0 : tune_layer.ws();
  for (const Layer& l : layers) ws_words = std::max(ws_words, l.ws());
  const size_t o_ws = take(sizeof(double2) * ws_words);
  const size_t o_ews = take(sizeof(double2) * 2 * BT_MAXCHI * BT_MAXCHI * std::max(1, nobs_total));
  std::vector<char> image(o_image_end - o_image, 0), results(o_results_end - o_results);  // (outlive the copies)
  char* base = nullptr;
  {
    cudaError_t e = cudaMallocAsync((void**)&base, off, s);
    if (e != cudaSuccess) return fail(QR_ENOMEM, std::string("batch state: ") + cudaGetErrorString(e));
  }
  struct MemGuard {
    void* p;
    cudaStream_t s;
    ~MemGuard() { cudaFreeAsync(p, s); cudaStreamSynchronize(s); }
  } mg{base, s};

  // ---- host image of the tables
  auto put = [&](size_t at, const void* src, size_t bytes) { memcpy(image.data() + (at - o_image), src, bytes); };
  std::vector<BTask> tasks;
  tasks.reserve(ntask_total);
  std::vector<size_t> layer_start(nlayers + 1, 0);
  for (int L = 0; L < nlayers; L++) {
    layer_start[L] = tasks.size();
    for (auto& qg : layer_tasks[L]) {
      const BReq& r = bt->reqs[qg.first];
      const ROff& o = ro[qg.first];
      const int s0 = r.gsite[qg.second];
      BTask t;
      t.sl = reinterpret_cast<double2*>(base + o.site[s0]);
      t.sr = reinterpret_cast<double2*>(base + o.site[s0 + 1]);
      t.lam = reinterpret_cast<double*>(base + o.lam[s0]);
      t.bd = reinterpret_cast<int*>(base + o.bd);
      t.haslam = reinterpret_cast<int*>(base + o.hl);
      t.gate = reinterpret_cast<const double2*>(base + o.gates) + 16 * qg.second;
      t.status = reinterpret_cast<int*>(base + o.status);
      t.threshold = r.threshold;
      t.bond = s0;
      t.nb = r.n - 1;
      t.maxdim = cap_of(r.n, s0, r.chi_max);
      t.pad = 0;
      tasks.push_back(t);
    }
  }
  layer_start[nlayers] = tasks.size();
  std::vector<BObs> obs;
  std::vector<double2*> sites_tab;
  for (int q = 0; q < R; q++) {
    const BReq& r = bt->reqs[q];
    const ROff& o = ro[q];
    std::vector<double2*> sp(r.n);
    std::vector<double*> lp(r.n - 1);
    for (int i = 0; i < r.n; i++) sp[i] = reinterpret_cast<double2*>(base + o.site[i]), sites_tab.push_back(sp[i]);
    for (int b = 0; b < r.n - 1; b++) lp[b] = reinterpret_cast<double*>(base + o.lam[b]);
    const std::vector<int> ones(r.n - 1, 1);
    const int ok = QR_OK;
    put(o.bd, ones.data(), sizeof(int) * (r.n - 1));  // (Lambda flags: zero)
    put(o.status, &ok, sizeof(int));
    put(o.sp, sp.data(), sizeof(double2*) * r.n);
    put(o.lp, lp.data(), sizeof(double*) * (r.n - 1));
    if (!r.gmat.empty()) put(o.gates, r.gmat.data(), sizeof(double2) * r.gmat.size());
    std::vector<int> pc((size_t)r.n * std::max<size_t>(1, r.ow.size()), 0);
    int pos = 0;
    for (size_t j = 0; j < r.ow.size(); j++) {
      for (int w = 0; w < r.ow[j]; w++, pos++) {
        // a repeated site multiplies its Paulis; strings come with distinct sites, later wins
        pc[(size_t)r.n * j + r.os[pos]] = r.op[pos];
      }
      BObs b;
      b.sites = reinterpret_cast<double2* const*>(base + o.sp);
      b.lams = reinterpret_cast<double* const*>(base + o.lp);
      b.bd = reinterpret_cast<const int*>(base + o.bd);
      b.haslam = reinterpret_cast<const int*>(base + o.hl);
      b.pauli = reinterpret_cast<const int*>(base + o.paulis) + (size_t)r.n * j;
      b.out = reinterpret_cast<double2*>(base + o.out) + j;
      b.n = r.n;
      b.pad = 0;
      obs.push_back(b);
    }
    put(o.paulis, pc.data(), sizeof(int) * pc.size());
  }
  if (!tasks.empty()) put(o_tasks, tasks.data(), sizeof(BTask) * tasks.size());
  if (!obs.empty()) put(o_obs, obs.data(), sizeof(BObs) * obs.size());
  put(o_sites_tab, sites_tab.data(), sizeof(double2*) * sites_tab.size());
  QR_CUDA(cudaMemcpyAsync(base + o_image, image.data(), image.size(), cudaMemcpyHostToDevice, s));

  double2* ws = reinterpret_cast<double2*>(base + o_ws);
  if (!bt->warps) QR_TRY(autotune(bt, s, key, tune_chi, tune_layer, ws));
  auto gate_kernel = (bt->precision & QR_MIXED) ? batch_gate_k<true> : batch_gate_k<false>;

  // ---- one CUDA graph: init, every layer, the expectation sweep
  const BTask* dtasks = reinterpret_cast<const BTask*>(base + o_tasks);
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  QR_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  int launches = 0;
  batch_init_k<<<std::max(1, std::min(1024, (nsites_total + 255) / 256)), 256, 0, s>>>(
      reinterpret_cast<double2* const*>(base + o_sites_tab), nsites_total);
  launches++;
  for (int L = 0; L < nlayers; L++) {
    const int nt = (int)(layer_start[L + 1] - layer_start[L]);
    if (nt == 0) continue;
    const Layer& l = layers[L];
    QR_CUDA(launch_cluster(gate_kernel, l.clusters, l.team, 32 * bt->warps, s, dtasks + layer_start[L], nt, ws, l.side, 0,
                           l.team));
    launches++;
  }
  if (!obs.empty()) {
    QR_CUDA(launch_cluster(batch_expect_k, (unsigned)obs.size(), BX_CL, BX_NT, s,
                           reinterpret_cast<const BObs*>(base + o_obs), reinterpret_cast<double2*>(base + o_ews)));
    launches++;
  }
  cudaError_t ce = cudaStreamEndCapture(s, &graph);
  if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
  struct GraphGuard {
    cudaGraph_t g;
    cudaGraphExec_t* x;
    ~GraphGuard() {
      if (*x) cudaGraphExecDestroy(*x);
      if (g) cudaGraphDestroy(g);
    }
  } gg{graph, &exec};
  QR_CUDA(cudaGraphInstantiate(&exec, graph, 0));
  size_t nodes = 0;
  QR_CUDA(cudaGraphGetNodes(graph, nullptr, &nodes));
  cudaEvent_t e0, e1;
  QR_CUDA(cudaEventCreate(&e0));
  QR_CUDA(cudaEventCreate(&e1));
  QR_CUDA(cudaEventRecord(e0, s));
  QR_CUDA(cudaGraphLaunch(exec, s));
  QR_CUDA(cudaEventRecord(e1, s));
  QR_CUDA(cudaEventSynchronize(e1));
  float gms = 0.f;
  QR_CUDA(cudaEventElapsedTime(&gms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  QR_CUDA(cudaGetLastError());
  count_launch((uint64_t)launches);
  bt->launches = launches;
  bt->layers = nlayers;
  bt->graph_nodes = nodes;
  bt->run_ms = gms;
  if (ms) *ms = gms;

  // ---- results
  QR_CUDA(cudaMemcpyAsync(results.data(), base + o_results, results.size(), cudaMemcpyDeviceToHost, s));
  QR_CUDA(cudaStreamSynchronize(s));
  auto get = [&](size_t at, void* dst, size_t bytes) { memcpy(dst, results.data() + (at - o_results), bytes); };
  for (int q = 0; q < R; q++) {
    BReq& r = bt->reqs[q];
    const ROff& o = ro[q];
    get(o.status, &r.status, sizeof(int));
    r.values.resize(r.ow.size());
    if (!r.ow.empty()) get(o.out, r.values.data(), sizeof(double2) * r.ow.size());
    r.bd.resize(r.n - 1);
    get(o.bd, r.bd.data(), sizeof(int) * (r.n - 1));
    std::vector<int> hl(r.n - 1);
    get(o.hl, hl.data(), sizeof(int) * (r.n - 1));
    r.lam.assign(r.n - 1, {});
    for (int b = 0; b < r.n - 1; b++) {
      if (!hl[b]) continue;
      r.lam[b].resize(r.bd[b]);
      get(o.lam[b], r.lam[b].data(), sizeof(double) * r.bd[b]);
    }
  }
  bt->ran = true;
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_result(const qr_batch* bt, int id, int* status, double* values) try {
  if (!bt || id < 0 || id >= (int)bt->reqs.size()) return fail(QR_EINVAL, "bad batch request id");
  if (!bt->ran) return fail(QR_EINVAL, "the batch has not run");
  const BReq& r = bt->reqs[id];
  if (status) *status = r.status;
  if (values)
    for (size_t j = 0; j < r.values.size(); j++) {
      values[2 * j] = r.values[j].x;
      values[2 * j + 1] = r.values[j].y;
    }
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_bond_dims(const qr_batch* bt, int id, int* out) try {
  if (!bt || id < 0 || id >= (int)bt->reqs.size()) return fail(QR_EINVAL, "bad batch request id");
  if (!bt->ran) return fail(QR_EINVAL, "the batch has not run");
  const BReq& r = bt->reqs[id];
  for (int b = 0; b < r.n - 1; b++) out[b] = r.bd[b];
  return QR_OK;
} QR_ABI_CATCH

int qr_batch_lambda(const qr_batch* bt, int id, int bond, double* out, int* len) try {
  if (!bt || id < 0 || id >= (int)bt->reqs.size()) return fail(QR_EINVAL, "bad batch request id");
  if (!bt->ran) return fail(QR_EINVAL, "the batch has not run");
  const BReq& r = bt->reqs[id];
  if (bond < 0 || bond >= r.n - 1) return fail(QR_EINVAL, "Invalid bond");
  if (len) *len = (int)r.lam[bond].size();
  if (out)
    for (size_t j = 0; j < r.lam[bond].size(); j++) out[j] = r.lam[bond][j];
  return QR_OK;
} QR_ABI_CATCH

// layers, kernel launches in the graph, graph nodes, warps per CTA chosen, 1 if the choice came
// from the tuning cache, graph time (ms), autotuning time (ms)
int qr_batch_info(const qr_batch* bt, int* layers, int* launches, int* graph_nodes, int* warps, int* cached,
                  double* run_ms, double* tune_ms) try {
  if (!bt) return fail(QR_EINVAL, "null batch");
  if (layers) *layers = bt->layers;
  if (launches) *launches = bt->launches;
  if (graph_nodes) *graph_nodes = (int)bt->graph_nodes;
  if (warps) *warps = bt->warps;
  if (cached) *cached = bt->tuned_from_cache;
  if (run_ms) *run_ms = bt->run_ms;
  if (tune_ms) *tune_ms = bt->tune_ms;
  return QR_OK;
} QR_ABI_CATCH

}  // extern "C"
