// Included by svd.cu: the finish of the Jacobi SVD by matrix products.
//
// From right singular vectors X (k x k) of FP32 quality, each step forms B = A X, G = B^H B and
// S = X^H X at FP64 accuracy on the tensor cores and corrects X <- X + X M, M = R / 2 + T + T^2 / 2:
// R = I - S restores unitarity and the anti-Hermitian T rotates all pairs that fail the Jacobi rotation
// test at once, T_pq = t g / |g| with the pair's Jacobi tangent t and the coupling
// g = G_pq + (l_p + l_q) R_pq / 2 that orthonormalised columns would have (l = diag G).  Tangents are
// squared from step to step (second-order terms of both corrections remain), so FP32 vectors
// (t ~ 1e-2) take three corrections and a final test.  A Jacobi sweep over 2048 columns is 1023
// dependent rounds, 72 ms in double-float; a step here is one and two half products of 2048^3, ~5 ms.
// The largest tangents (near-degenerate clusters) go through a listed double-float Jacobi sweep instead, which is
// never the last word: the next step forms B = A X again and corrects X, so results carry FP64 and not 48 bits.
// (Ogita and Aishima, "Iterative refinement for symmetric eigenvalue decomposition", 2018, give the first-order form
// of the correction.)

// The pairs of the first step within this factor of its largest tangent, and at any step those at or
// above kRefineListTan, are left out of T and rotated by a listed sweep: the second-order terms of the rest
// fall with the square.
constexpr float kRefineListFrac = 0.5f, kRefineListTan = 0.04f;
// Bound of |T|_2 for a simultaneous rotation; beyond it the steps would not contract.
constexpr float kRefineMaxNorm = 0.5f;
// A column whose tangents sum to more than this meets more large ones than a list should order.
constexpr float kRefineCrowd = 4.f;
// A step whose second-order terms, bounded by the largest tangent and |R| times the largest column sums,
// are below this part of the tolerance needs no further test.
constexpr float kRefineLast = 0.03f;
constexpr int kRefineMaxSteps = 12;
// Couplings that meet the tolerance are turned along with the others, down to a sixteenth of it, where that takes a
// tangent of at most this.  Left alone they add up: |U S V^H - A| of 512 x 512 in FP64 is 18 - 23 eps sigma_max over
// flat, linear and twofold to fourfold degenerate spectra instead of 106 - 227.  Their second-order terms are this part of
// couplings below the tolerance, so no test waits for them; larger tangents would show the products' 2^-23.
constexpr float kRefineTidyTan = 1e-7f;

// Column q of T per block: the rotation test of the pairs (p, q) and T_pq (diagonal 0).  out[0] += pairs
// (p < q) that fail the test, out[1] = their largest tangent, out[2] = largest |R|, out[3] = largest sum of
// their tangents in a column, out[5] = of all tangents in a column, a bound of |T|_2 (float bits).
__global__ void __launch_bounds__(256) refine_pairs_k(const double2* __restrict__ G, const double2* __restrict__ S, int k,
                                                      int k0, double tol, const double* __restrict__ smax_p,
                                                      double2* __restrict__ T, unsigned* __restrict__ out) {
  __shared__ float red[8][4];
  __shared__ unsigned redc[8];
  const double smax = smax_p[0] / smax_p[1];
  const float fl = (float)(4.0 * Eps<double>::v * smax);
  const float tols = (float)(tol * smax);
  const int q = blockIdx.x;
  const double lq = G[(long)q * (k + 1)].x;
  unsigned cnt = 0;
  float tmax = 0.f, rmax = 0.f, sum = 0.f, all = 0.f;
  for (int p = threadIdx.x; p < k; p += 256) {
    const long e = p + (long)q * k;
    const double2 s = S[e];
    double2 t = make_double2(0.0, 0.0);
    if (p == q) {
      rmax = fmaxf(rmax, fabsf((float)(1.0 - s.x)));
    } else {
      rmax = fmaxf(rmax, fmaxf(fabsf((float)s.x), fabsf((float)s.y)));
      if (min(p, q) < k0) {
        const double lp = G[(long)p * (k + 1)].x;
        const double h = 0.5 * (lp + lq);
        const double2 g0 = G[e];
        const float gx = (float)(g0.x - h * s.x), gy = (float)(g0.y - h * s.y);
        const float big = fmaxf(fabsf(gx), fabsf(gy));
        // scaled magnitude: squares of tiny couplings would underflow
        const float inv = big > 0.f ? 1.f / big : 0.f;
        const float ux = gx * inv, uy = gy * inv, un = sqrtf(ux * ux + uy * uy), g = big * un;
        const float lim = tols * sqrtf((float)fmin(lp, lq)) + fl * fl;
        if (lp > 0.0 && lq > 0.0 && g > 0.0625f * lim) {
          const float d = (float)(lq - lp);
          const float az = fabsf(d) / (2.f * g);
          const float tt = az > 1e18f ? 0.5f / az : 1.f / (az + sqrtf(1.f + az * az));
          // equal norms: the sign of a zero difference must differ between T_pq and T_qp
          const float sg = ((d < 0.f || (d == 0.f && p > q)) ? -tt : tt) / un;
          const bool fails = g > lim;
          if (fails || tt <= kRefineTidyTan) {
            t = make_double2((double)(sg * ux), (double)(sg * uy));
            all += tt;
          }
          if (fails) {
            if (p < q) cnt++;
            tmax = fmaxf(tmax, tt);
            sum += tt;
          }
        }
      }
    }
    T[e] = t;
  }
  for (int o = 16; o > 0; o >>= 1) {
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
    rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    all += __shfl_xor_sync(0xffffffffu, all, o);
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[w][0] = tmax;
    red[w][1] = rmax;
    red[w][2] = sum;
    red[w][3] = all;
    redc[w] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; i++) {
      tmax = fmaxf(tmax, red[i][0]);
      rmax = fmaxf(rmax, red[i][1]);
      sum += red[i][2];
      all += red[i][3];
      cnt += redc[i];
    }
    if (cnt) atomicAdd(out, cnt);
    atomicMax(out + 1, __float_as_uint(tmax));
    atomicMax(out + 2, __float_as_uint(rmax));
    atomicMax(out + 3, __float_as_uint(sum));
    atomicMax(out + 5, __float_as_uint(all));
  }
}

// Marks the pairs with |T_pq| >= thr in the list (vertices of `width` columns) and takes them out of T.
__global__ void refine_mark_k(double2* __restrict__ T, int k, float thr, int width, unsigned* ml, int nv) {
  const MaskedList L = masked_list(ml, nv);
  const long tot = (long)k * k;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
    const int p = (int)(e % k), q = (int)(e / k);
    const double2 t = T[e];
    const float x = (float)t.x, y = (float)t.y;
    if (x * x + y * y < thr * thr) continue;
    T[e] = make_double2(0.0, 0.0);
    if (p > q) continue;
    const int vp = p / width, vq = q / width;
    if (vp == vq) L.flag[vp] = 1u;
    else atomicOr(L.mask + (long)vp * L.mw + (vq >> 5), 1u << (vq & 31));
  }
}

// T <- M = (I - S) / 2 + T + T2 / 2 (T2 may be null)
__global__ void refine_m_k(double2* __restrict__ T, const double2* __restrict__ T2, const double2* __restrict__ S, int k) {
  const long tot = (long)k * k;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
    const double2 s = S[e];
    double2 m = T[e];
    if (T2) {
      const double2 u = T2[e];
      m.x += 0.5 * u.x;
      m.y += 0.5 * u.y;
    }
    m.x += 0.5 * ((e % k == e / k ? 1.0 : 0.0) - s.x);
    m.y -= 0.5 * s.y;
    T[e] = m;
  }
}
// T <- the first-order correction that makes unit columns with Gram matrix S orthonormal: a pair's overlap is taken
// from its columns in the shares sigma_p^2 and sigma_q^2 that move U diag(sigma) least
__global__ void orthonormal_m_k(double2* __restrict__ T, const double2* __restrict__ S, const double* __restrict__ sigma,
                                int k) {
  const long tot = (long)k * k;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
    const long p = e % k, q = e / k;
    const double2 s = S[e];
    const float r = sigma[p] > 0.0 ? (float)(sigma[q] / sigma[p]) : 1e18f;
    const float w = -1.f / (1.f + r * r);  // column p's share in column q
    T[e] = p == q ? make_double2(0.5 * (1.0 - s.x), 0.0) : make_double2(w * s.x, w * s.y);
  }
}
// L (m x k, ld ldl) += Y (ld m)
__global__ void add_cols_k(double2* __restrict__ L, long ldl, const double2* __restrict__ Y, int m, int k) {
  const long tot = (long)m * k;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < tot; e += (long)gridDim.x * blockDim.x) {
    double2* d = L + e % m + e / m * ldl;
    d->x += Y[e].x;
    d->y += Y[e].y;
  }
}
__global__ void add_to_k(double2* __restrict__ X, const double2* __restrict__ Y, long n) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    X[e].x += Y[e].x;
    X[e].y += Y[e].y;
  }
}

// One double-float Jacobi sweep over the pairs marked in w->ml (vertices of `width` columns: 2, the
// block sweep, or 1, the scalar sweep) on the FP64 arrays B = A X (rows x k) and X (k x k).
int df_listed(cudaStream_t s, SvdWork* w, double2* B, int rows, int k, double2* X, int width, int nv, double tol,
              const double* smax_d, int k0, long* listed) {
  const size_t kk = (size_t)k * k, rk = (size_t)rows * k;
  int classes = 0;
  QR_TRY(upload_schedule(s, w, nv, true, listed, &classes));
  if (*listed == 0) return QR_OK;
  QR_TRY(w->Bl.ensure(sizeof(float2) * 2 * rk, s));
  QR_TRY(w->Rm.ensure(sizeof(float2) * 2 * kk, s));
  float2 *Bh = w->Bl.as<float2>(), *Bl = Bh + rk, *Xh = w->Rm.as<float2>(), *Xl = Xh + kk;
  QR_TRY(z2df(s, B, rows, rows, k, nullptr, Bh, Bl, rows));
  QR_TRY(z2df(s, X, k, k, k, nullptr, Xh, Xl, k));
  const int nstate = 8 + SW_STRIDE;
  QR_TRY(w->cnt.ensure(sizeof(unsigned) * (nstate + nv + 16), s));
  unsigned *state = w->cnt.as<unsigned>(), *done = state + nstate;
  QR_CUDA(cudaMemsetAsync(state, 0, sizeof(unsigned) * (nstate + nv), s));
  int sms = 0, per_sm = 0, kz = k0, sw = 0, mm = rows, kk2 = k, nvv = nv;
  long l1 = rows, l2 = k;
  unsigned* fl = nullptr;
  unsigned* mlp = w->ml.as<unsigned>();
  QR_TRY(device_sm_count(&sms));
  int pr = prof_begin(s, PK_JACOBI_DF, 0.0, 0.0);
  if (width == 2) {
    const size_t sm = sizeof(float2) * 8 * (size_t)k;
    QR_TRY(set_func_attr_once((const void*)jacobi_block_df_k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(sizeof(float2) * 8 * DB_MAXROWS)));
    QR_TRY(blocks_per_sm((const void*)jacobi_block_df_k, DB_NT, sm, &per_sm));
    if (per_sm < 1) return fail(QR_ECUDA, "double-float block sweep kernel cannot be resident");
    svd_path(SP_DF_BLOCK);
    void* args[] = {&Bh, &Bl, &l1, &mm, &kk2, &Xh, &Xl, &l2, &nvv, &tol, &smax_d, &state, &sw, &fl, &kz, &mlp, &done};
    QR_CUDA(cudaLaunchCooperativeKernel((const void*)jacobi_block_df_k, dim3(std::max(1, std::min(per_sm * sms, nv / 2))),
                                        dim3(DB_NT), args, sm, s));
  } else {
    const size_t sm = (k % 2 == 0 && k <= 4096) ? sizeof(float2) * 4 * (size_t)k : 0;
    const void* f = (const void*)jacobi_sweep_df_k<256, 8>;
    QR_TRY(set_func_attr_once(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(float2) * 4 * 4096));
    QR_TRY(blocks_per_sm(f, 256, sm, &per_sm));
    if (per_sm < 1) return fail(QR_ECUDA, "double-float sweep kernel cannot be resident");
    svd_path(SP_DF_DATAFLOW);
    void* args[] = {&Bh, &Bl, &l1, &mm, &kk2, &Xh, &Xl, &l2, &nvv, &tol, &smax_d, &state, &sw, &fl, &kz, &mlp, &done};
    QR_CUDA(cudaLaunchCooperativeKernel(f, dim3(std::max(1, std::min(per_sm * sms, nv / 2))), dim3(256), args, sm, s));
  }
  count_launch();
  prof_end(s, pr);
  svd_path(SP_DF_MASKED);
  QR_TRY(df2z(s, Xh, Xl, k, k, k, nullptr, X, k));
  QR_TRY(df2z(s, Bh, Bl, rows, rows, k, nullptr, B, rows));
  unsigned* hs = static_cast<unsigned*>(host_scratch(sizeof(unsigned) * nstate));
  if (!hs) return fail(QR_ENOMEM, "page-locked host scratch");
  QR_CUDA(cudaMemcpyAsync(hs, state, sizeof(unsigned) * nstate, cudaMemcpyDeviceToHost, s));
  QR_CUDA(cudaStreamSynchronize(s));
  if (hs[4]) return fail(QR_ECUDA, "double-float Jacobi sweep: a column wait timed out");
  float tmax;
  memcpy(&tmax, &hs[9], sizeof(float));
  if (debug_on())
    fprintf(stderr, "[qr] refine %dx%d: listed sweep of %ld pairs of %d-column blocks in %d classes: %u rotations, max tan %.2e\n",
            rows, k, *listed, width, classes, hs[8], tmax);
  prof_account(pr, 96.0 * rows * (width == 2 ? 4.0 : 1.0) * *listed + 344.0 * hs[8] * (rows + k),
               sizeof(float2) * 4.0 * ((double)rows + k) * (*listed + hs[8]), 1);
  return QR_OK;
}

// X (k x k, ld k, in and out) and B = A X (rows x k, ld rows; A may not alias it) such that no pair with
// a column below k0 fails the rotation test of tolerance `tol`.  *done = 0: the steps do not converge; X
// is unitary and B = A X, from which the caller finishes with sweeps.
int refine(cudaStream_t s, SvdWork* w, const double2* A, int rows, int k, double2* X, double2* B, double tol,
           const double* smax_d, int k0, int* done) {
  const size_t kk = (size_t)k * k;
  const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
  *done = 0;
  QR_TRY(w->rfG.ensure(sizeof(double2) * 3 * kk, s));
  double2 *G = w->rfG.as<double2>(), *S = G + kk, *T = S + kk;
  // listed sweeps: pairs of 2-column blocks in registers, or single pairs; none for the cluster sizes
  const int width = rows <= DB_MAXROWS && k % 2 == 0 ? 2 : 1;
  const int nv0 = (k + width - 1) / width, nv = nv0 + (nv0 & 1);
  const bool lists = k > 128 && nv < 32768;
  if (lists) QR_TRY(w->ml.ensure(sizeof(unsigned) * masked_list_words(nv), s));
  QR_TRY(w->rfc.ensure(64, s));
  unsigned* out = w->rfc.as<unsigned>();
  const bool tc = k >= 192;  // small products: the FP64-accurate kernels have the lower latency
  unsigned* err = out + 4;
  void* tcw = nullptr;
  if (tc) {
    QR_TRY(w->tcw.ensure(zgemm_tc_workspace(k, k, k, 1, true), s));
    tcw = w->tcw.as<char>();
  }
  auto product = [&](const double2* P, const double2* Q2, double2* C) {
    return tc ? zgemm_tc(s, OP_N, OP_N, k, k, k, P, k, 0, Q2, k, 0, C, k, 0, 1, tcw, err)
              : zgemm(s, OP_N, OP_N, k, k, k, one, P, k, 0, Q2, k, 0, zero, C, k, 0, 1, nullptr, true);
  };
  unsigned* hs = static_cast<unsigned*>(host_scratch(sizeof(unsigned) * 8));
  if (!hs) return fail(QR_ENOMEM, "page-locked host scratch");
  QR_CUDA(cudaMemsetAsync(out, 0, 32, s));
  float last = 1e30f;
  bool pending = false;  // marked pairs wait for the next B = A X
  int lists_run = 0;
  bool give_up = false;  // only the unitary correction from here on, for the caller's sweeps
  for (int step = 0; step < kRefineMaxSteps + 8; step++) {
    give_up = give_up || step >= kRefineMaxSteps;
    QR_TRY(zgemm_graded(s, rows, k, k, A, rows, X, k, B, rows));
    const bool swept = pending;  // B and X have been through double-float: one more step before they are results
    if (pending) {
      long listed = 0;
      QR_TRY(df_listed(s, w, B, rows, k, X, width, nv, 32.0 * sqrt((double)rows) * Eps<double>::v, smax_d, k0, &listed));
      pending = false;
      lists_run++;
    }
    QR_TRY(zherk(s, k, rows, B, rows, G, k));
    QR_TRY(zherk(s, k, k, X, k, S, k));
    QR_CUDA(cudaMemsetAsync(out, 0, 16, s));
    QR_CUDA(cudaMemsetAsync(out + 5, 0, 4, s));
    refine_pairs_k<<<k, 256, 0, s>>>(G, S, k, k0, tol, smax_d, T, out);
    QR_CHECK_LAUNCH("refine_pairs_k");
    hs = static_cast<unsigned*>(host_scratch(sizeof(unsigned) * 8));
    if (!hs) return fail(QR_ENOMEM, "page-locked host scratch");
    QR_CUDA(cudaMemcpyAsync(hs, out, 32, cudaMemcpyDeviceToHost, s));
    QR_CUDA(cudaStreamSynchronize(s));
    if (hs[4]) return fail(QR_ECUDA, "tcgen05 product: a bounded wait gave up");
    const unsigned fail_pairs = hs[0];
    float tmax, rmax, tsum, tall;
    memcpy(&tmax, &hs[1], sizeof(float));
    memcpy(&rmax, &hs[2], sizeof(float));
    memcpy(&tsum, &hs[3], sizeof(float));
    memcpy(&tall, &hs[5], sizeof(float));
    if (debug_on())
      fprintf(stderr, "[qr] refine %dx%d step %d: %u pairs, largest tangent %.2e, column sum %.2e; |I - X^H X| %.2e\n", rows,
              k, step, fail_pairs, tmax, tsum, rmax);
    if (!(rmax < 0.5f) || !(tmax <= 1.f)) return fail(QR_ENOCONV, "SVD refinement: vectors far from unitary");
    if (rmax < 1e-14f && !swept && (fail_pairs == 0 || give_up)) {
      *done = give_up ? 0 : 1;
      return QR_OK;
    }
    bool rotate = fail_pairs > 0 && !give_up;
    if (rotate && (lists && (tmax >= kRefineListTan || step == 0))) {
      // list the large tangents; with too many of them (degenerate clusters) nothing rotates until X is
      // unitary, and the caller's sweeps take over if that does not separate them
      const float thr = step == 0 ? kRefineListFrac * fmaxf(tmax, kRefineListTan * 0.01f) : kRefineListTan;
      const bool crowded = tsum > kRefineCrowd || lists_run >= 4;
      if (!crowded) {
        unsigned* ml = w->ml.as<unsigned>();
        const MaskedList L = masked_list(ml, nv);
        QR_CUDA(cudaMemsetAsync(ml, 0, sizeof(unsigned) * (size_t)(L.items - L.mask), s));
        refine_mark_k<<<gs((long)kk), TPB, 0, s>>>(T, k, fminf(thr, kRefineListTan), width, ml, nv);
        QR_CHECK_LAUNCH("refine_mark_k");
        pending = true;
      } else {
        rotate = false;
        give_up = rmax < 1e-9f;
      }
    } else if (rotate && tsum > kRefineMaxNorm) {
      rotate = false;
      give_up = rmax < 1e-9f;
    }
    if (rmax < 1e-9f && rotate && !pending) {
      if (tmax > 0.5f * last) {
        rotate = false;
        give_up = true;
      }
      last = tmax;
    }
    const bool second = rotate && tall > 1e-8f;
    if (rotate) svd_path(SP_DF_LINEAR);
    else QR_CUDA(cudaMemsetAsync(T, 0, sizeof(double2) * kk, s));
    if (second) QR_TRY(product(T, T, G));
    refine_m_k<<<gs((long)kk), TPB, 0, s>>>(T, second ? G : nullptr, S, k);
    QR_CHECK_LAUNCH("refine_m_k");
    QR_TRY(product(X, T, G));
    add_to_k<<<gs((long)kk), TPB, 0, s>>>(X, G, (long)kk);
    QR_CHECK_LAUNCH("add_to_k");
    if (!give_up && !pending && (rotate || fail_pairs == 0) && tmax * tsum <= kRefineLast * (float)tol &&
        rmax * (tsum + rmax) <= kRefineLast * (float)tol) {
      QR_TRY(zgemm_graded(s, rows, k, k, A, rows, X, k, B, rows));
      if (tc) {
        QR_CUDA(cudaMemcpyAsync(hs, err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        QR_CUDA(cudaStreamSynchronize(s));
        if (hs[0]) return fail(QR_ECUDA, "tcgen05 product: a bounded wait gave up");
      }
      *done = 1;
      return QR_OK;
    }
  }
  return fail(QR_ENOCONV, "SVD refinement: the vectors do not become unitary");
}
