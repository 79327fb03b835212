// Included by svd.cu: FP32 block Jacobi sweeps whose block pairs are diagonalised through their Gram matrix
// (gram_item.cuh).

// One sweep: clusters of cs CTAs take the items (round, pair) in order, ordered by per-block flags as
// jacobi_sweep_dev_k's columns are.  A wait that gives up sets state[4] / state[5] and the sweep runs on
// without waiting (its result is discarded), so that no CTA leaves while others read its shared memory.
template <int W, int NT>
__global__ void __launch_bounds__(NT, NT == 128 ? 4 : 2)
    jacobi_gram_k(float2* __restrict__ B, long ldb, int m, int n, float2* __restrict__ V, long ldv, int nbp, float tol,
                  const double* __restrict__ smax_p, unsigned* __restrict__ state, int sweep, unsigned* __restrict__ flags,
                  float tan_stop, int cs) {
  extern __shared__ __align__(16) float2 gr_rows[];
  __shared__ GrShared<W> sh;
  if (((volatile unsigned*)state)[0]) return;
  const float smax = (float)(smax_p[0] / smax_p[1]);
  unsigned* cnt = state + 8 + SW_STRIDE * sweep;
  const int nb = (n + W - 1) / W, npairs = nbp / 2, rank = blockIdx.x % cs, ncl = gridDim.x / cs;
  const unsigned base = (unsigned)sweep * (unsigned)(nbp - 1);
  const long total = (long)(nbp - 1) * npairs;
  for (long it = blockIdx.x / cs; it < total; it += ncl) {
    const int round = (int)(it / npairs), pair = (int)(it % npairs);
    int bp, bq;
    pair_cols(nbp, round, pair, bp, bq);
    wait_cols(flags, bp, bq, nb, base + round, state);
    // (a block that meets the padding block only has pairs in round 0)
    if (bq < nb || round == 0)
      gr_item<W, NT>(B, ldb, m, n, V, ldv, nb, bp, bq, round == 0, tol, smax, cnt, sh, gr_rows, rank * NT, rank, cs);
    if (cs > 1) {  // every CTA's stores precede the flags; and the partial Gram matrices have been read
      __syncwarp();
      cluster_sync_all();
    }
    if (rank == 0) post_cols(flags, bp, bq, nb, base + round + 1);
    else __syncthreads();
  }
  finish_sweep(state, cnt, sweep, tan_stop);
}

// Up to 128 columns and 128 rows: all sweeps in one cluster, a CTA per item of a round, the cluster barrier
// between rounds.  state as in jacobi_cluster_k.
template <int W>
__global__ void __launch_bounds__(JC_NT) jacobi_gram_cluster_k(float2* __restrict__ B, long ldb, int m, int n,
                                                               float2* __restrict__ V, long ldv, float tol,
                                                               const double* __restrict__ smax_p, int max_sweeps,
                                                               unsigned* __restrict__ state, float tan_stop) {
  extern __shared__ __align__(16) float2 gr_rows[];
  __shared__ GrShared<W> sh;
  const float smax = (float)(smax_p[0] / smax_p[1]);
  const int nb = (n + W - 1) / W, nbp = nb + (nb & 1), npairs = nbp / 2;
  int sweep = 0;
  bool conv = false;
  for (; sweep < max_sweeps && !conv; sweep++) {
    unsigned* cnt = state + 8 + SW_STRIDE * sweep;
    for (int round = 0; round < nbp - 1; round++) {
      for (int pair = blockIdx.x; pair < npairs; pair += gridDim.x) {
        int bp, bq;
        pair_cols(nbp, round, pair, bp, bq);
        if (bq < nb || round == 0) 
          gr_item<W, JC_NT>(B, ldb, m, n, V, ldv, nb, bp, bq, round == 0, tol, smax, cnt, sh, gr_rows, 0, 0, 1);
        __syncthreads();  // shared state is reused by the next item
      }
      cluster_sync_all();
    }
    const unsigned h = __ldcg(cnt);
    const float tmax = __uint_as_float(__ldcg(cnt + 1));
    conv = h == 0 || tmax < tan_stop;
    cluster_sync_all();  // everyone has read this sweep's counters
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    state[0] = conv ? 1u : 0u;
    state[1] = sweep;
  }
}

constexpr int GR_MAXROWS = 16 * 256;  // 16 CTAs of 256 rows

// resident clusters of a kernel at a cluster size, cached per device
int resident_clusters(const void* f, int threads, int cs, const cudaLaunchConfig_t& cfg, int* out) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, int>, int> known;
  int dev = 0;
  QR_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_tuple(dev, f, threads, cs);
  auto it = known.find(key);
  if (it == known.end()) {
    int v = 0;
    QR_CUDA(cudaOccupancyMaxActiveClusters(&v, f, &cfg));
    it = known.emplace(key, v).first;
  }
  *out = it->second;
  return QR_OK;
}

// The launch of one full sweep over k columns of up to GR_MAXROWS rows (the larger of rows and k): block
// width, rows per CTA, cluster size and grid.
struct GramPlan {
  const void* kernel = nullptr;
  int W = 16, NT = 256, cs = 1, nbp = 0, grid = 0;
  size_t smem = 0;
};
void gram_config(const GramPlan& g, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, cudaStream_t s) {
  cfg->gridDim = dim3(g.grid);
  cfg->blockDim = dim3(g.NT);
  cfg->dynamicSmemBytes = g.smem;
  cfg->stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = g.cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;  // the flag waits need every cluster resident
  attr[1].val.cooperative = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 2;
}
int gram_plan(int rows, int k, GramPlan* g) {
  const int r = std::max(rows, k);
  // Wide blocks once L2 traffic and not the rounds' latency bounds a sweep, and several CTAs per item in
  // between (ms per sweep at W, NT = 8,256 / 8,128 / 16,256: 256 columns 0.35 0.37 0.46, 512 0.83 0.77 0.99,
  // 768 1.59 1.43 1.52, 1024 2.20 2.23 2.03, 2048 15.6 18.0 11.0)
  g->W = r <= 896 ? 8 : 16;
  g->NT = r <= 256 || r > 896 ? 256 : 128;
  if (g->W == 16) {
    g->kernel = (const void*)jacobi_gram_k<16, 256>;
    g->smem = gr_smem<16, 256>();
  } else {
    g->kernel = g->NT == 256 ? (const void*)jacobi_gram_k<8, 256> : (const void*)jacobi_gram_k<8, 128>;
    g->smem = g->NT == 256 ? gr_smem<8, 256>() : gr_smem<8, 128>();
  }
  g->cs = (r + g->NT - 1) / g->NT;
  const int nb = (k + g->W - 1) / g->W;
  g->nbp = nb + (nb & 1);
  QR_TRY(set_func_attr_once(g->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g->smem));
  if (g->cs > 8) QR_TRY(set_func_attr_once(g->kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  gram_config(*g, &cfg, attr, nullptr);
  cfg.gridDim = dim3(g->cs);
  cfg.numAttrs = 1;
  int resident = 0;
  QR_TRY(resident_clusters(g->kernel, g->NT, g->cs, cfg, &resident));
  if (resident < 1) return fail(QR_ECUDA, "block Jacobi sweep clusters cannot be resident");
  g->grid = std::min(resident, g->nbp / 2) * g->cs;
  return QR_OK;
}
