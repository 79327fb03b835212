// The SVD of one small matrix (up to 128 x 128) on one thread-block cluster: FP32 Jacobi sweeps, then their
// rotations refined by products until they diagonalise the matrix to rounding.  Shared by the SVD (svd.cu) and
// the batched engine's gate step (batch.cu).
#pragma once
#include "common.cuh"
#include "jacobi_rot.cuh"
#include "gram_item.cuh"

namespace qr {
namespace {

constexpr int TM_MAXK = 128;  // rows and columns

// Every phase is dealt to the cluster's threads or warps, and the data goes through L2.  `Team` is this
// thread's place in the cluster.
struct Team {
  int size, rank;       // CTAs, this CTA
  int tid, nt;          // thread of the cluster, its threads
  int lane, warp, nw;   // warp of the cluster, its warps
  __device__ __forceinline__ void sync() const {
    if (size == 1) {
      __syncthreads();
    } else {
      __syncwarp();
      cluster_sync_all();
    }
  }
};

// Rotations and largest tangent of a sweep, counted by the whole team: sweep s uses slot s % 3 and clears
// the next one, which was last read two barriers ago.
struct SweepCount {
  unsigned* c;  // 3 x 2 words in global memory
  __device__ __forceinline__ void start(const Team& T) const {
    if (T.tid == 0) { __stcg(c, 0u); __stcg(c + 1, 0u); }
  }
  __device__ __forceinline__ unsigned* open(const Team& T, int sweep) const {
    unsigned* nx = c + 2 * ((sweep + 1) % 3);
    if (T.tid == 0) { __stcg(nx, 0u); __stcg(nx + 1, 0u); }
    return c + 2 * (sweep % 3);
  }
  static __device__ __forceinline__ void add(unsigned* s, float tabs) {
    atomicAdd(s, 1u);
    atomicMax(s + 1, __float_as_uint(tabs));
  }
  static __device__ __forceinline__ bool done(const unsigned* s, float tan_stop) {
    return __ldcg(s) == 0u || __uint_as_float(__ldcg(s + 1)) < tan_stop;
  }
};

// pair `pair` of round `round` over np (even) columns, p < q
__device__ __forceinline__ void round_pair(int np, int round, int pair, int& p, int& q) {
  if (pair == 0) { p = round; q = np - 1; }
  else { p = (round + pair) % (np - 1); q = (round - pair + np - 1) % (np - 1); }
  if (p > q) { const int x = p; p = q; q = x; }
}

constexpr int TM_RPL = TM_MAXK / 32;  // rows a lane

// FP64 Hestenes sweeps of the team on B (rows x k, ld rows) accumulating V (k x k, ld k): round-robin pairs,
// one warp per pair with the columns' rows in registers, a team barrier between rounds.  Stops after a sweep
// that rotates nothing or whose largest rotation tangent is below tan_stop; returns that verdict.
__device__ bool team_sweeps(const Team& T, double2* B, double2* V, int rows, int k, double tol, double smax,
                            int max_sweeps, float tan_stop, SweepCount cnt) {
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
        double2 *bp = B + (long)rows * p, *bq = B + (long)rows * q, *vp = V + (long)k * p, *vq = V + (long)k * q;
        double2 x[TM_RPL], y[TM_RPL], u[TM_RPL], w[TM_RPL];
        double a = 0, bb = 0, gr = 0, gi = 0;
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          const int r = T.lane + 32 * j;
          x[j] = y[j] = u[j] = w[j] = make_double2(0.0, 0.0);
          if (r < rows) { x[j] = __ldcg(bp + r); y[j] = __ldcg(bq + r); }
          if (r < k) { u[j] = __ldcg(vp + r); w[j] = __ldcg(vq + r); }
        }
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          if (32 * j >= rows) break;  // no arithmetic on rows that no lane has
          a += x[j].x * x[j].x + x[j].y * x[j].y;
          bb += y[j].x * y[j].x + y[j].y * y[j].y;
          gr += x[j].x * y[j].x + x[j].y * y[j].y;
          gi += x[j].x * y[j].y - x[j].y * y[j].x;
        }
        a = warp_sum(a); bb = warp_sum(bb); gr = warp_sum(gr); gi = warp_sum(gi);
        double c, sr, si;
        float tabs;
        if (!rotation_params<double>(a, bb, gr, gi, tol, smax, c, sr, si, tabs)) continue;
#pragma unroll
        for (int j = 0; j < TM_RPL; j++) {
          const int r = T.lane + 32 * j;
          if (32 * j < rows) {
            rot(x[j], y[j], c, sr, si);
            if (r < rows) { __stcg(bp + r, x[j]); __stcg(bq + r, y[j]); }
          }
          if (32 * j < k) {
            rot(u[j], w[j], c, sr, si);
            if (r < k) { __stcg(vp + r, u[j]); __stcg(vq + r, w[j]); }
          }
        }
        if (T.lane == 0) SweepCount::add(sc, tabs);
      }
      T.sync();
    }
    converged = SweepCount::done(sc, tan_stop);
  }
  T.sync();  // the counters have been read
  return converged;
}

// FP32 sweeps on Gram matrices of block pairs (gram_item.cuh), an item a CTA; up to TM_MAXK rows.
constexpr int TM_W = 8;
constexpr size_t TM_TILE = gr_smem<TM_W, TM_MAXK>() / sizeof(float2);
constexpr float TM_STOP32 = 0.15f;  // tangent of the last FP32 sweep: what is left is second order in it
__device__ void team_sweeps_f32(const Team& T, float2* B, float2* V, int rows, int k, float tol, float smax,
                                int max_sweeps, float tan_stop, SweepCount cnt, GrShared<TM_W>& sh, float2* tile) {
  const int nb = (k + TM_W - 1) / TM_W, nbp = nb + (nb & 1), npairs = nbp / 2;
  bool converged = false;
  cnt.start(T);
  T.sync();
  for (int sweep = 0; sweep < max_sweeps && !converged; sweep++) {
    unsigned* sc = cnt.open(T, sweep);
    for (int round = 0; round < nbp - 1; round++) {
      for (int pair = T.rank; pair < npairs; pair += T.size) {
        int bp, bq;
        round_pair(nbp, round, pair, bp, bq);
        if (bq < nb || round == 0) {
          if (threadIdx.x < TM_MAXK)
            gr_item<TM_W, TM_MAXK>(B, rows, rows, k, V, k, nb, bp, bq, round == 0, tol, smax, sc, sh, tile, 0, 0, 1);
        }
        __syncthreads();  // shared state is reused by the next item
      }
      T.sync();
    }
    converged = SweepCount::done(sc, tan_stop);
  }
  T.sync();  // the counters have been read
}

// ---- the refinement ----------------------------------------------------------------------------------
__device__ __forceinline__ void mac(double2& s, double2 a, double2 b) {
  s.x = fma(a.x, b.x, fma(-a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(a.y, b.x, s.y));
}
__device__ __forceinline__ void macc(double2& s, double2 a, double2 b) {  // conj(a) b
  s.x = fma(a.x, b.x, fma(a.y, b.y, s.x));
  s.y = fma(a.x, b.y, fma(-a.y, b.x, s.y));
}
// the sum of `parts` neighbouring lanes
__device__ __forceinline__ double2 parts_sum(double2 s, int parts) {
  for (int o = 1; o < parts; o <<= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  return s;
}

// lanes that share one sum: as many as the team has threads for, so that a small product is not one chain of
// k dependent multiply-adds
__device__ __forceinline__ int team_parts(const Team& T, int sums) {
  int p = 1;
  while (p < 8 && 2 * p * sums <= T.nt) p *= 2;
  return p;
}

// Ct[i + k r] = sum_x A[r, x] Xt[i + k x]: A rows x k (ld rows), X k x k and C rows x k by rows
__device__ void team_product(const Team& T, double2* A, int rows, double2* Xt, int k, double2* Ct) {
  const int parts = team_parts(T, rows * k), total = rows * k * parts;
  for (int t0 = T.tid - T.lane; t0 < total; t0 += T.nt) {
    const int t = t0 + T.lane, part = t % parts, e = t / parts, i = e % k, r = e / k;
    double2 s = make_double2(0.0, 0.0);
    if (t < total) {
#pragma unroll 2
      for (int x = part; x < k; x += parts) mac(s, A[r + rows * x], Xt[i + k * x]);
    }
    s = parts_sum(s, parts);
    if (t < total && part == 0) Ct[e] = s;
  }
}

// G = B^H B and S = X^H X - I for B (rows x k) and X (k x k) by rows: half of each, column i with column i - d.
// gs[i + k j] = (G_ij, S_ij) of the computed pairs, dg[i] = G_ii, gs[i + k i].z = S_ii.
__device__ void team_grams(const Team& T, double2* Bt, int rows, double2* Xt, int k, float4* gs, double* dg) {
  const int sums = k * (k / 2 + 1), parts = team_parts(T, sums), total = sums * parts;
  for (int t0 = T.tid - T.lane; t0 < total; t0 += T.nt) {
    const int t = t0 + T.lane, part = t % parts, e = t / parts, i = e % k, d = e / k, j = i >= d ? i - d : i - d + k;
    const bool on = t < total && !(2 * d == k && i < j);  // (the other end of an opposite pair has it)
    double2 g = make_double2(0.0, 0.0), s = make_double2(d == 0 && part == 0 ? -1.0 : 0.0, 0.0);
    if (on) {
#pragma unroll 2
      for (int r = part; r < rows; r += parts) macc(g, Bt[i + k * r], Bt[j + k * r]);
#pragma unroll 2
      for (int x = part; x < k; x += parts) macc(s, Xt[i + k * x], Xt[j + k * x]);
    }
    const double2 gv = parts_sum(g, parts), sv = parts_sum(s, parts);
    if (on && part == 0) {
      gs[i + k * j] = make_float4((float)gv.x, (float)gv.y, (float)sv.x, (float)sv.y);
      if (d == 0) dg[i] = gv.x;
    }
  }
}

constexpr float TM_BIGTAN = 0.03f;   // tangents above this are not rotated at once
constexpr float TM_LASTTAN = 1e-8f;  // a correction this small leaves nothing above rounding
// Couplings that meet the tolerance are turned too, down to a sixteenth of it, where that takes a rotation this
// small: a step forms them anyway, and left alone they add up in the factors.
constexpr float TM_TIDYTAN = 1e-9f;
constexpr int TM_STEPS = 10;

// The correction E of X <- X + X E, Et[i + k j] = E[j, i]: -S / 2, and for a pair that fails the rotation test
// of rotation_params (or may be tidied up) its tangent times the phase of its coupling, as orthonormal columns would
// have it.  count[1] <- largest |E| of the former, count[0] += tangents above TM_BIGTAN (left out).
__device__ inline void team_correction(const Team& T, const float4* gs, const double* dg, int k, double tol, double smax,
                                       bool rotate, float2* Et, unsigned* count) {
  const double fl = 4.0 * Eps<double>::v * smax, t2 = tol * tol * smax * smax, fl4 = fl * fl * fl * fl;
  unsigned big = 0;
  float emax = 0.f;
  for (int e = T.tid; e < k * (k / 2 + 1); e += T.nt) {
    const int i = e % k, d = e / k, j = i >= d ? i - d : i - d + k;
    if (2 * d == k && i < j) continue;
    const float4 v = gs[i + k * j];
    const float rx = -0.5f * v.z, ry = -0.5f * v.w;
    emax = fmaxf(emax, fmaxf(fabsf(rx), fabsf(ry)));
    if (d == 0) {
      Et[i + k * i] = make_float2(rx, 0.f);
      continue;
    }
    const double a = dg[i], b = dg[j], h = 0.5 * (a + b);
    const double gx = v.x - h * v.z, gy = v.y - h * v.w, g2 = gx * gx + gy * gy;
    float sx = 0.f, sy = 0.f;
    const double lim = t2 * fmin(a, b) + fl4;
    if (rotate && a > 0.0 && b > 0.0 && g2 > lim * (1.0 / 256.0)) {
      // (the coupling may lie below FP32's range)
      const float big_g = (float)fmax(fabs(gx), fabs(gy));
      const float inv = 1.f / big_g, ux = (float)gx * inv, uy = (float)gy * inv, ru = rsqrtf(ux * ux + uy * uy);
      const float z = (float)(0.5 * (b - a)) * inv * ru, tt = (z >= 0.f ? 1.f : -1.f) / (fabsf(z) + sqrtf(1.f + z * z));
      const bool fails = g2 > lim;
      if (fails && fabsf(tt) > TM_BIGTAN) {
        big++;
      } else if (fails || fabsf(tt) <= TM_TIDYTAN) {
        sx = tt * ux * ru;
        sy = tt * uy * ru;
        if (fails) emax = fmaxf(emax, fabsf(tt));
      }
    }
    Et[j + k * i] = make_float2(rx + sx, ry + sy);   // E[i, j] = s
    Et[i + k * j] = make_float2(rx - sx, -ry + sy);  // E[j, i] = -conj(s)
  }
  big = __reduce_add_sync(0xffffffffu, big);
  const unsigned em = __reduce_max_sync(0xffffffffu, __float_as_uint(emax));
  if (T.lane == 0) {
    if (big) atomicAdd(count, big);
    atomicMax(count + 1, em);
  }
}

// Yt = (X + X E)^T: FP32 products of X's FP32 values Xf, |E| < TM_BIGTAN
__device__ void team_correct(const Team& T, double2* Xt, const float2* Xf, const float2* Et, int k,
                             double2* Yt) {
  const int parts = team_parts(T, k * k), total = k * k * parts;
  for (int t0 = T.tid - T.lane; t0 < total; t0 += T.nt) {
    const int t = t0 + T.lane, part = t % parts, e = t / parts, i = e % k, x = e / k;
    float re = 0.f, im = 0.f;
    if (t < total) {
#pragma unroll 4
      for (int j = part; j < k; j += parts) {
        const float2 a = Xf[j + k * x], b = Et[i + k * j];
        re = fmaf(a.x, b.x, fmaf(-a.y, b.y, re));
        im = fmaf(a.x, b.y, fmaf(a.y, b.x, im));
      }
    }
    for (int o = 1; o < parts; o <<= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (t < total && part == 0) Yt[e] = make_double2(Xt[e].x + re, Xt[e].y + im);
  }
}

// B (rows x k, ld rows) = the columns of Bt (by rows) made orthogonal: b_q -= b_p g / (d_p + d_q) and b_p -= b_q
// conj(g) / (d_p + d_q) with g = b_p^H b_q, d the squared norms (dg), the least change of B that does it.  B = A X
// rounds every column at eps smax, which is eps smax / sigma of a short one: a product's columns over 3 decades are
// 100 to 1000 eps from orthogonal, after this 10.
__device__ void team_tidy(const Team& T, double2* Bt, int rows, int k, const double* dg, double2* G, double2* B) {
  const int sums = k * (k - 1) / 2, parts = team_parts(T, sums), total = sums * parts;
  for (int t0 = T.tid - T.lane; t0 < total; t0 += T.nt) {
    const int t = t0 + T.lane, part = t % parts, e = t / parts;
    int q = (int)((sqrtf(8.f * e + 1.f) + 1.f) * 0.5f);  // e = q (q - 1) / 2 + p, p < q
    while (q * (q - 1) / 2 > e) q--;
    while ((q + 1) * q / 2 <= e) q++;
    const int p = e - q * (q - 1) / 2;
    double2 s = make_double2(0.0, 0.0);
    if (t < total) {
#pragma unroll 2
      for (int r = part; r < rows; r += parts) macc(s, Bt[p + k * r], Bt[q + k * r]);
    }
    s = parts_sum(s, parts);
    if (t < total && part == 0) {
      const float d = (float)dg[p] + (float)dg[q], inv = d > 1e-30f ? 1.f / d : 0.f;
      const double2 c = make_double2(s.x * inv, s.y * inv);
      G[p + k * q] = c;
      G[q + k * p] = cconj(c);
    }
  }
  T.sync();
  const int nb = rows * k, pb = team_parts(T, nb), tb = nb * pb;
  for (int t0 = T.tid - T.lane; t0 < tb; t0 += T.nt) {
    const int t = t0 + T.lane, part = t % pb, e = t / pb, j = e % k, r = e / k;
    double2 s = make_double2(0.0, 0.0);
    if (t < tb) {
#pragma unroll 2
      for (int i = part; i < k; i += pb)
        if (i != j) mac(s, Bt[i + k * r], G[i + k * j]);
    }
    s = parts_sum(s, pb);
    if (t < tb && part == 0) B[r + rows * j] = csub(Bt[j + k * r], s);
  }
}

// Squares of side^2 double2 that team_svd works in, and one column (norms, sweep counters).
constexpr int TM_SQUARES = 7;
constexpr size_t team_ws(int side) { return TM_SQUARES * (size_t)side * side + TM_MAXK; }

// Right singular vectors V (k x k, ld k) of A (rows x k, ld rows; scaled: largest column norm smax in [1/2, 1))
// and B = A V (A's own place or another), whose columns are orthogonal to tol smax min(|b_p|, |b_q|).
//
// FP32 sweeps on a copy of A (64x the FP64 rate) leave rotations X of FP32 quality; each step then forms
// B = A X, B^H B and X^H X and corrects X to first order, which squares what is left: two or three steps.  If
// pairs need a large rotation still (columns far below smax, whose couplings the absolute FP32 test leaves), FP32
// sweeps with a relative test run once more on B, and if that does not do, full-precision sweeps finish.
//
// A Jacobi sweep is a chain of k - 1 rounds, each with the latency of a dozen dependent FP64 operations: ~5000
// cycles a round.  A step is four phases.
__device__ bool team_svd(const Team& T, double2* A, double2* B, double2* V, int rows, int k, double tol, double smax,
                         double2* ws, int side, GrShared<TM_W>& sh, float2* tile) {
  const size_t K2 = (size_t)side * side;
  double2 *S0 = ws, *S1 = ws + K2, *S2 = S1 + K2, *S3 = S2 + K2, *S4 = S3 + K2, *S5 = S4 + K2, *S6 = S5 + K2;
  double2* tail = S6 + K2;
  double* dg = reinterpret_cast<double*>(tail);
  const SweepCount cnt{reinterpret_cast<unsigned*>(dg + TM_MAXK)};
  float2 *B32 = reinterpret_cast<float2*>(S0), *V32 = B32 + K2;
  double2 *Am = S1, *X = S2, *Y = S3, *Bt = S4;
  float4* gs = reinterpret_cast<float4*>(S5);
  float2* Et = reinterpret_cast<float2*>(S6);
  for (int t = T.tid; t < rows * k; t += T.nt) {
    const double2 v = A[t];
    B32[t] = make_float2((float)v.x, (float)v.y);
    Am[t] = v;
  }
  for (int t = T.tid; t < k * k; t += T.nt) V32[t] = make_float2(t % k == t / k ? 1.f : 0.f, 0.f);
  const float tol32 = fmaxf(4e-6f, 2.f * sqrtf((float)rows) * Eps<float>::v);
  team_sweeps_f32(T, B32, V32, rows, k, tol32, (float)smax, 20, TM_STOP32, cnt, sh, tile);
  for (int t = T.tid; t < k * k; t += T.nt) X[t / k + k * (t % k)] = make_double2(V32[t].x, V32[t].y);
  cnt.start(T);
  T.sync();
  bool again = false, rotate = true, done = false;
  for (int step = 0; step < TM_STEPS && !done; step++) {
    team_product(T, Am, rows, X, k, Bt);
    T.sync();
    team_grams(T, Bt, rows, X, k, gs, dg);
    for (int t = T.tid; t < k * k; t += T.nt) V32[t] = make_float2((float)X[t].x, (float)X[t].y);
    unsigned* c = cnt.open(T, step);
    T.sync();
    team_correction(T, gs, dg, k, tol, smax, rotate, Et, c);
    T.sync();
    const unsigned big = __ldcg(c);
    const float emax = __uint_as_float(__ldcg(c + 1));
    if (big && !again) {
      again = true;
      for (int t = T.tid; t < rows * k; t += T.nt) B32[t / k + rows * (t % k)] = make_float2((float)Bt[t].x, (float)Bt[t].y);
      for (int t = T.tid; t < k * k; t += T.nt) V32[t] = make_float2(t % k == t / k ? 1.f : 0.f, 0.f);
      T.sync();
      team_sweeps_f32(T, B32, V32, rows, k, -tol32, (float)smax, 20, TM_STOP32, cnt, sh, tile);
      for (int t = T.tid; t < k * k; t += T.nt) {  // X <- X V32
        const int i = t % k, x = t / k;
        double2 s = make_double2(0.0, 0.0);
        for (int j = 0; j < k; j++) mac(s, X[j + k * x], make_double2(V32[j + k * i].x, V32[j + k * i].y));
        Y[t] = s;
      }
      double2* z = X; X = Y; Y = z;
      cnt.open(T, step);  // (the next step's counters)
      T.sync();
      continue;
    }
    if (big && rotate) {  // only make X unitary from here on
      rotate = false;
      T.sync();
      continue;
    }
    team_correct(T, X, V32, Et, k, Y);
    T.sync();
    double2* z = X; X = Y; Y = z;
    done = emax <= TM_LASTTAN;
  }
  // X is unitary and diagonalises, or is the start of full sweeps (the identity, if it did not become unitary)
  if (done) {
    team_product(T, Am, rows, X, k, Bt);
    T.sync();
    for (int t = T.tid; t < k * k; t += T.nt) V[t] = X[t % k * k + t / k];
    if (rotate) team_tidy(T, Bt, rows, k, dg, reinterpret_cast<double2*>(S5), B);
    else for (int t = T.tid; t < rows * k; t += T.nt) B[t] = Bt[t % rows * k + t / rows];
  } else {
    for (int t = T.tid; t < rows * k; t += T.nt) B[t] = A[t];
    for (int t = T.tid; t < k * k; t += T.nt) V[t] = make_double2(t % k == t / k ? 1.0 : 0.0, 0.0);
  }
  T.sync();
  if (done && rotate) return true;
  return team_sweeps(T, B, V, rows, k, tol, smax, 60, 1e-8f, cnt);
}
// column norms of B (rows x k, ld rows) into nrm (global), and into every CTA's sig after the barrier
__device__ void team_norms(const Team& T, const double2* B, int rows, int k, double* nrm, double* sig) {
  for (int j = T.warp; j < k; j += T.nw) {
    double s = 0.0;
    for (int r = T.lane; r < rows; r += 32) {
      const double2 v = B[r + (long)rows * j];
      s += v.x * v.x + v.y * v.y;
    }
    s = warp_sum(s);
    if (T.lane == 0) __stcg(nrm + j, sqrt(s));
  }
  T.sync();
  for (int j = threadIdx.x; j < k; j += blockDim.x) sig[j] = __ldcg(nrm + j);
  __syncthreads();
}


}  // namespace
}  // namespace qr
