// FP32 rotations of a pair of column blocks found on their Gram matrix: the work item of the block Jacobi
// sweeps of the SVD (svd_gram.cuh) and of the batched engine's gate step (batch.cu).
//
// The k columns form blocks of W; a work item is a pair of blocks, 2 W columns.  Its CTAs (a cluster of cs,
// one row per thread) form the 2 W x 2 W Gram matrix of the columns once, rotate the item's pairs on that
// matrix in shared memory (W rounds of W disjoint cross pairs; in round 0 of a sweep, where every block
// appears once, 2 W - 1 rounds of all pairs), and then apply the recorded rotations to their rows of B and V,
// which stay in registers.  Every CTA of a cluster sums the same partial Gram matrices in the same order, so
// all of them find the same rotations.
//
// Forming each local round's inner products from the rows instead (as the listed sweeps do) costs a reduction
// over the rows per round and, at 4 columns a block, 5.3 TB/s of L2 traffic at 2048 columns.  That sweep took
// 0.66 ms at 256 columns (now 0.35), 1.5 at 512 (0.77), 3.4 at 1024 (2.0), 12.6 at 2048 (11.0), and the whole
// FP32 stage of a 128 x 128 block 1.57 ms (0.95).  An item of 32 columns x 256 rows spends a fifth of its time
// each on the Gram matrix, the rotations of B and those of V, a quarter on the Gram rotations (~900 cycles a
// round, one dependent chain) and the rest on loads, sums and the cluster's exchanges.  The rotated Gram matrix
// carries FP32 rounding relative to the column norms, like the inner products it replaces.
//
// The item's pairs move through fixed register positions: position i of the first half meets position i of
// the second, and after each round the columns shift (cross rounds: the second half by one; all pairs: the
// circle method), so the rotation code is one unrolled round whose registers need no dynamic index.
#pragma once
#include "common.cuh"
#include "jacobi_rot.cuh"

namespace qr {
namespace {

// position of the first half (0 .. W - 1) or second half (W .. 2 W - 1) after the shift that ends a round
template <int W>
__device__ __forceinline__ int gr_next(bool full, int x) {
  if (!full) return x < W ? x : W + (x - W + W - 1) % W;
  if (x < W) return x == 0 ? 0 : x < W - 1 ? x + 1 : 2 * W - 1;
  return x == W ? 1 : x - 1;
}

template <int W>
struct GrShared {
  float2 G[2][2 * W * (2 * W + 1)];                  // by position, rows of 2 W + 1
  float4 rot[(2 * W - 1) * W];                       // (c, s_re, s_im, tangent) of round r, position i: [r W + i]
  float2 part[(W / 2) * (W / 2 + 1) / 2 * 16];       // this CTA's partial Gram matrix, 4 x 4 tiles
  unsigned count, tmax;
};
template <int W, int NT>
constexpr size_t gr_smem() { return sizeof(float2) * NT * (2 * W + 2); }

// Rotation of the pair with squared norms a, b and product g (the test of rotation_params_f32), from the
// normalised product g / (|x| |y|) so that small columns do not underflow; c and s by fast approximations
// and one Newton step for c (the vectors' loss of unitarity is the sum of its errors).  c = 1, s = 0 when
// the pair stays.
struct GrRot {
  float c, sr, si, t;
};
__device__ __forceinline__ float gr_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ GrRot gr_params(float a, float b, float2 g, float tol, float smax) {
  // (a zero column gives infinities and NaN, and fails the test)
  const float ra = gr_rsqrt(a), rb = gr_rsqrt(b);
  const float ur = (g.x * ra) * rb, ui = (g.y * ra) * rb, u2 = ur * ur + ui * ui;
  const float fl = 4.f * Eps<float>::v * smax, fa = (fl * ra) * (fl * ra), fb = (fl * rb) * (fl * rb);
  const float tr = tol * smax * fminf(ra, rb);
  const float thr = tol < 0.f ? tol * tol : tr * tr + fa * fb;
  const bool go = a > 1e-37f && b > 1e-37f && u2 > thr;
  // cot(2 theta) = |z|: with r = sin(2 theta), c^2 = (1 + |z| r) / 2 and s = r / (2 c)
  const float ru = gr_rsqrt(u2);
  const float z = 0.5f * ((b * ra) * rb - (a * ra) * rb) * ru;
  const float az = fminf(fabsf(z), 1e9f), r = gr_rsqrt(1.f + az * az);
  const float c2 = 0.5f + 0.5f * az * r;
  float ic = gr_rsqrt(c2);
  ic = ic * (1.5f - 0.5f * c2 * ic * ic);
  const float s = 0.5f * r * ic;
  const float e = (z < 0.f ? -s : s) * ru;
  GrRot p;
  p.c = go ? c2 * ic : 1.f;
  p.sr = go ? e * ur : 0.f;
  p.si = go ? e * ui : 0.f;
  p.t = go ? s * ic : 0.f;
  return p;
}

// the warps that rotate on the Gram matrix, and those that work on the item (the first NT threads of a CTA)
template <int N>
__device__ __forceinline__ void gr_inner_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void gr_item_sync() {
  asm volatile("bar.sync 2, %0;" ::"n"(N) : "memory");
}

// rotations of one recorded round on a row, then the shift
template <int W>
__device__ __forceinline__ void gr_round(float2 (&x)[2 * W], const float4* rot_r, bool full) {
#pragma unroll
  for (int i = 0; i < W; i++) {
    const float4 p = rot_r[i];  // pairs that stay carry the identity: no branch between the loads
    rot(x[i], x[W + i], p.x, p.y, p.z);
  }
  if (!full) {
    const float2 t = x[W];
#pragma unroll
    for (int i = 0; i < W - 1; i++) x[W + i] = x[W + i + 1];
    x[2 * W - 1] = t;
  } else {
    const float2 last = x[W - 1], b0 = x[W];
#pragma unroll
    for (int i = W - 1; i > 1; i--) x[i] = x[i - 1];
    x[1] = b0;
#pragma unroll
    for (int i = 0; i < W - 1; i++) x[W + i] = x[W + i + 1];
    x[2 * W - 1] = last;
  }
}

// One work item: blocks bp < bq of nb; this CTA's first NT threads hold rows row0 + tid of B (m rows) and V (n
// rows).
template <int W, int NT>
__device__ __forceinline__ void gr_item(float2* __restrict__ B, long ldb, int m, int n, float2* __restrict__ V, long ldv,
                                        int nb, int bp, int bq, bool full, float tol, float smax, unsigned* cnt,
                                        GrShared<W>& sh, float2* rows, int row0, int rank, int cs) {
  constexpr int C = 2 * W, LD = C + 2, TC = C / 4, NTL = TC * (TC + 1) / 2, NG = NT / NTL;
  static_assert(NG >= 1 && NG * NTL * 16 <= NT * LD, "the group sums reuse the row tile");
  const int tid = threadIdx.x, r = row0 + tid;
  const int nq = min(W, n - bq * W);  // bq may be the padding block (bq >= nb: no columns)
  const int np = min(W, n - bp * W);
  auto colp = [&](int c) { return c < W ? (c < np ? bp * W + c : -1) : (bq < nb && c - W < nq ? bq * W + c - W : -1); };
  if (tid == 0) sh.count = sh.tmax = 0;
  float2 x[C];
#pragma unroll
  for (int c = 0; c < C; c++) {
    const int col = colp(c);
    x[c] = (col >= 0 && r < m) ? __ldcg(B + (long)col * ldb + r) : make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int c = 0; c < C; c += 2)
    *reinterpret_cast<float4*>(rows + tid * LD + c) = make_float4(x[c].x, x[c].y, x[c + 1].x, x[c + 1].y);
  gr_item_sync<NT>();
  // partial Gram matrix: a thread owns a 4 x 4 tile on or above the diagonal for every NG-th row
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.f, 0.f);
  const int g = tid / NTL, tl = tid % NTL;
  int tj = 0;
  while ((tj + 1) * (tj + 2) / 2 <= tl) tj++;
  const int ti = tl - tj * (tj + 1) / 2;
  const int live = min(NT, max(0, m - row0));
  if (g < NG) {
#pragma unroll 2
    for (int q = g; q < live; q += NG) {
      const float4* ra = reinterpret_cast<const float4*>(rows + q * LD + 4 * ti);
      const float4* rb = reinterpret_cast<const float4*>(rows + q * LD + 4 * tj);
      const float4 a0 = ra[0], a1 = ra[1], b0 = rb[0], b1 = rb[1];
      const float2 a[4] = {{a0.x, a0.y}, {a0.z, a0.w}, {a1.x, a1.y}, {a1.z, a1.w}};
      const float2 b[4] = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}, {b1.z, b1.w}};
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          acc[i][j].x += a[i].x * b[j].x + a[i].y * b[j].y;
          acc[i][j].y += a[i].x * b[j].y - a[i].y * b[j].x;
        }
    }
  }
  gr_item_sync<NT>();
  if (g < NG) {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) rows[(g * 16 + 4 * i + j) * NTL + tl] = acc[i][j];
  }
  gr_item_sync<NT>();
  for (int e = tid; e < NTL * 16; e += NT) {
    float2 s = rows[e];
    for (int q = 1; q < NG; q++) s = cadd(s, rows[q * 16 * NTL + e]);
    sh.part[e] = s;
  }
  if (cs > 1) {
    __syncwarp();
    cluster_sync_all();
  } else {
    gr_item_sync<NT>();
  }
  for (int e = tid; e < NTL * 16; e += NT) {
    const int t2 = e % NTL, ij = e / NTL;
    int j2 = 0;
    while ((j2 + 1) * (j2 + 2) / 2 <= t2) j2++;
    const int p = 4 * (t2 - j2 * (j2 + 1) / 2) + ij / 4, q = 4 * j2 + ij % 4;
    if (p > q) continue;
    float2 s = sh.part[e];
    if (cs > 1) {
      s = make_float2(0.f, 0.f);
      for (int c = 0; c < cs; c++) {
        uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(&sh.part[e])), ra;
        float2 v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(c));
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(ra) : "memory");
        s = cadd(s, v);
      }
    }
    if (p == q) s.y = 0.f;
    sh.G[0][p * (C + 1) + q] = s;
    sh.G[0][q * (C + 1) + p] = make_float2(s.x, -s.y);
  }
  gr_item_sync<NT>();
  // Rotations on the Gram matrix, G <- J^H G J per round: the first warp forms the rotations and the
  // pairs' own blocks, the next ones update the 2 x 2 blocks of pairs (a, b), a < b, a thread each.  G is kept
  // by position and written to the positions after the shift, so a thread's addresses are the same in every
  // round.  A round is one dependent chain (~900 cycles): only the warps that take part synchronise in it.
  const int nr = full ? 2 * W - 1 : W;
  constexpr int NBL = W * (W - 1) / 2, GR_INNER = 32 + (NBL + 31) / 32 * 32, LG = C + 1;
  constexpr int PART = GR_INNER <= NT ? GR_INNER : NT, SLOTS = (NBL + PART - 33) / (PART - 32);
  if (tid < PART) {
    unsigned count = 0;
    float tmax = 0.f;
    int a_[SLOTS], b_[SLOTS], wr[SLOTS][4];
#pragma unroll
    for (int u = 0; u < SLOTS; u++) {
      const int q = tid - 32 + u * (PART - 32);
      int b = 1;
      while ((b + 1) * b / 2 <= q) b++;
      b_[u] = tid >= 32 && q < NBL ? b : -1;
      a_[u] = q - b * (b - 1) / 2;
      wr[u][0] = gr_next<W>(full, a_[u]);
      wr[u][1] = gr_next<W>(full, W + a_[u]);
      wr[u][2] = gr_next<W>(full, b);
      wr[u][3] = gr_next<W>(full, W + b);
    }
    const int dt = gr_next<W>(full, tid % W), db = gr_next<W>(full, W + tid % W);
    for (int rd = 0; rd < nr; rd++) {
      const float2* G = sh.G[rd & 1];
      float2* N = sh.G[(rd & 1) ^ 1];
      GrRot p = {1.f, 0.f, 0.f, 0.f};
      float d = 0.f, e = 0.f;
      float2 g = make_float2(0.f, 0.f);
      if (tid < W) {
        const float2* ta = G + tid * LG;
        d = ta[tid].x;
        e = ta[W * LG + W + tid].x;
        g = ta[W + tid];
        p = gr_params(d, e, g, tol, smax);
        sh.rot[rd * W + tid] = make_float4(p.c, p.sr, p.si, p.t);
      }
      gr_inner_sync<PART>();
      if (tid < W) {
        count += p.t > 0.f;
        tmax = fmaxf(tmax, p.t);
        // a rotated pair is diagonal, with squared norms d -+ tan(theta) |g|
        const float h = p.t > 0.f ? (e >= d ? -p.t : p.t) * sqrtf(g.x * g.x + g.y * g.y) : 0.f;
        const float2 o = p.t > 0.f ? make_float2(0.f, 0.f) : g;
        N[dt * LG + dt] = make_float2(d + h, 0.f);
        N[db * LG + db] = make_float2(e - h, 0.f);
        N[dt * LG + db] = o;
        N[db * LG + dt] = make_float2(o.x, -o.y);
      }
#pragma unroll
      for (int u = 0; u < SLOTS; u++) {
        if (b_[u] < 0) continue;
        const int a = a_[u], b = b_[u], wta = wr[u][0], wba = wr[u][1], wtb = wr[u][2], wbb = wr[u][3];
        const float2 *ta = G + a * LG, *ba = ta + W * LG;
        float2 m00 = ta[b], m01 = ta[W + b], m10 = ba[b], m11 = ba[W + b];
        const float4 j1 = sh.rot[rd * W + a], j2 = sh.rot[rd * W + b];
        // block (rows of pair a; columns of pair b): columns first ([x' y'] = [x y] J2), then rows (J1^H)
        rot(m00, m01, j2.x, j2.y, j2.z);
        rot(m10, m11, j2.x, j2.y, j2.z);
        // rows: conj(x) transforms as x does
        m00.y = -m00.y; m01.y = -m01.y; m10.y = -m10.y; m11.y = -m11.y;
        rot(m00, m10, j1.x, j1.y, j1.z);
        rot(m01, m11, j1.x, j1.y, j1.z);
        // the values are conjugated: they belong to the mirrored entries
        N[wtb * LG + wta] = m00; N[wta * LG + wtb] = make_float2(m00.x, -m00.y);
        N[wbb * LG + wta] = m01; N[wta * LG + wbb] = make_float2(m01.x, -m01.y);
        N[wtb * LG + wba] = m10; N[wba * LG + wtb] = make_float2(m10.x, -m10.y);
        N[wbb * LG + wba] = m11; N[wba * LG + wbb] = make_float2(m11.x, -m11.y);
      }
      gr_inner_sync<PART>();
    }
    if (count) {
      atomicAdd(&sh.count, count);
      atomicMax(&sh.tmax, __float_as_uint(tmax));
    }
  }
  gr_item_sync<NT>();
  if (sh.count == 0) return;
  if (tid == 0 && rank == 0) {
    atomicAdd(cnt, sh.count);
    atomicMax(cnt + 1, sh.tmax);
  }
#pragma unroll 1
  for (int rd = 0; rd < nr; rd++) gr_round<W>(x, sh.rot + rd * W, full);
#pragma unroll
  for (int c = 0; c < C; c++) {
    const int col = colp(c);
    if (col >= 0 && r < m) __stcg(B + (long)col * ldb + r, x[c]);
  }
  if (r < n) {
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int col = colp(c);
      x[c] = col >= 0 ? __ldcg(V + (long)col * ldv + r) : make_float2(0.f, 0.f);
    }
#pragma unroll 1
    for (int rd = 0; rd < nr; rd++) gr_round<W>(x, sh.rot + rd * W, full);
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int col = colp(c);
      if (col >= 0) __stcg(V + (long)col * ldv + r, x[c]);
    }
  }
}

}  // namespace
}  // namespace qr
