// FP64 complex GEMM on the Blackwell tensor cores: C[b] = op(A[b]) diag(dk) op(B[b]), the operands cut
// into seven 8-bit integer slices whose products are exact (the splitting of Ozaki, Ogita, Oishi and
// Rump, "Error-free transformations of matrix multiplication", 2012, with fixed slice widths).
//
// This part runs FP64 at ~1.1 TFLOP/s (DMMA and DFMA alike; 7 GFLOP/s per SM), 1/1700 of its BF16 rate,
// so the whole product is done in integers held as BF16:
//  1. oz_kmax_k: g_k = exponent of the largest entry of row k of op(B).  op(A)'s column k is scaled by
//     2^g_k and op(B)'s row k by 2^-g_k (exact), so a sum over k whose operands grade in opposite
//     directions (a Gamma tensor's 1/lambda against an environment's lambda) keeps its small terms.
//  2. oz_digits_k: row i of op(A) and column j of op(B) are scaled by powers of two E_i, E_j so that all
//     entries are below 1/2, rounded to 55-bit fixed point and written as seven signed bytes,
//     v = sum_s q_s 2^(8 (6 - s)), as BF16 planes, K-major.  The entry within a binade of the maximum is
//     exact; the rest are rounded at 2^-54 of it (an FP64 product rounds each sum instead).  A is
//     real-ified, [[Ar, -Ai], [Ai, Ar]], in 128-row tiles of 64 complex rows.  Integer and FP32
//     instructions only.
//  3. zgemm_oz_k: the 28 slice products with i + j = d <= 6 as tcgen05.mma (M 128, N 64, K 16) into
//     seven TMEM accumulators, one per d (448 of 512 columns, which is why the tile is 64 columns wide; the
//     guard below takes the rest).  Each |q q'| <= 2^14, so a sum of 256 k' stays below 2^24 for d <= 3 and every FP32 addition there
//     is exact; d >= 4 weighs at most 2^-32 of the leading sum and stays exact while its sums, random in
//     sign, are below 2^24 (2^19 after 1024 k' of random bytes).  The accumulators of d <= 3 are drained
//     every 256 k', those of d >= 4 every 1024, into two 64-bit integers per element, while the other
//     group's products keep the tensor core busy.  Neither the K order nor the split of K over a cluster
//     changes a bit of an exact sum (with the guard d = 6 rounds, see there).  The epilogue rounds hi + lo once to FP64.
// The first neglected products (d = 7) lie at 2^-56 of the row and column maxima (with the guard, below, 2^-64).
// Rows or columns that hold an infinity or NaN are recomputed by plain FP64 dot products in the epilogue.
// So the error is relative to the maxima of a row and a column, and an element whose products are all far below
// them (entries over many decades, the large ones of the row against the small ones of the column) would lose
// digits that an FP64 product keeps.  With the guard an eighth accumulator sums the products of the leading
// bytes' absolute values, sum |a||b| in units of 2^-14 of the two maxima, and elements where it is below
// OZ_LEAST sqrt(K) are formed in FP64 instead, a warp each.  The guard also adds the products of d = 7, whose absence is
// the larger part of the error where a row's maximum stands out (R's diagonal: R diag(Lambda) B at 256 columns is
// 1.0e-15 off without and 2.0e-16 with them, an FP64 product 7e-16): with slice s weighed 2^(-8 s), which bf16 holds
// exactly, they go into the accumulator of d = 6, whose sums then round at 2^-24 of themselves, 2^-66 of the maxima.
// What is left is the rounding of the entries.  Measured over entries exp(2 x) and exp(6 x) (x normal), 12 decades,
// 2% nonzeros and K of 64 to 4096, relative to sum |a||b|: rms 0.2 - 9e-16, largest 0.4 - 9e-15 (without the guard up
// to 7e-7 and 1e-4; an FP64 product 1 - 8e-15 at the largest).  A line four times lower doubles that, and a line twice
// as high takes 1.8 ms instead of 1.1 where every other element is one term (an orthogonal 1024 x 1024 factor with noise
// for zeros, times 1024 x 2048; 0.75 for ordinary entries).  Products whose error the caller needs relative to norms
// only (orthogonal factors, refinement, QR updates) do without.
//
// Bound: the MMAs, 28 products x 2 per 32 k' (about 51 cycles each: at N = 64 shared memory feeds the
// tensor core 6 KB per MMA in 48; with the guard 35 x 2); loads alone take 60% of that.  The kernel alone at 2048^3:
// 1.80 ms (38 TFLOP/s complex-equivalent, FP64 DMMA 1.06), 2.06 with the guard, tensor pipe 46 and 50% busy, its
// operand ports in shared memory 69 and 75%.  All three launches: 2.09 and 2.36 ms; at 512^3 77 and 84 us, at
// 256 x 512 x 256 47 and 49, most of it launches and the latency of one tile.  A tile grid that would leave SMs idle splits K over a cluster of up to 8 CTAs, which add
// their integer sums through distributed shared memory.
#include <cuda_bf16.h>
#include <algorithm>
#include <climits>
#include <map>
#include <tuple>
#include "kernels.cuh"
#include "prof.cuh"
#include "tcgen05.cuh"

namespace qr {

namespace {

constexpr int OZ_S = 7;                       // slices per operand
constexpr int OZ_BM = 128, OZ_BN = 64;        // output tile: 64 complex rows (re, im) x 64 columns
constexpr int OZ_BK = 32;                     // k' per stage (64-byte bf16 rows)
constexpr int OZ_STAGES = 2;
// Drains of the two accumulator groups, in stages: d <= 3 ("H") after stages 7, 15, ..., d >= 4 ("L") after
// stages 3, 35, 67, ..., and both after the last one.
constexpr int OZ_DH = 4;                      // accumulators of H
__device__ __forceinline__ bool oz_drain_h(int n, int last) { return n % 8 == 7 || n == last; }
__device__ __forceinline__ bool oz_drain_l(int n, int last) { return n % 32 == 3 || n == last; }
constexpr int OZ_AT = OZ_BM * OZ_BK * 2, OZ_BT = OZ_BN * OZ_BK * 2;  // bytes of one slice tile
// with the guard an eighth plane: the leading bytes' absolute values
constexpr int oz_planes(bool guard) { return OZ_S + (guard ? 1 : 0); }
constexpr int oz_stage(bool guard) { return oz_planes(guard) * (OZ_AT + OZ_BT); }
constexpr int OZ_EPI_WARPS = 16;              // four per TMEM lane quarter, 16 columns each
constexpr int OZ_THREADS = 32 * (2 + OZ_EPI_WARPS);  // warp 0 TMA, warp 1 MMA + TMEM, then the drain
constexpr int oz_smem(bool guard) { return OZ_STAGES * oz_stage(guard) + 1024 + 256; }
constexpr int OZ_TMEM_COLS = 512;
// after the products the stage memory holds the integer sums and, with the guard, its sums and a list of elements
constexpr int OZ_SUMS = OZ_BM * OZ_BN * 16, OZ_GSUMS = OZ_BM * OZ_BN * 4, OZ_LIST = 16 + 64 * OZ_BN * 2;
static_assert(OZ_SUMS <= OZ_STAGES * oz_stage(false), "the integer sums reuse the stage memory");
static_assert(OZ_SUMS + OZ_GSUMS + OZ_LIST <= OZ_STAGES * oz_stage(true), "so do the guard's");
static_assert(oz_smem(true) <= 227 * 1024, "two stages of eight planes");
constexpr int OZ_BAD = INT_MIN;               // exponent of a row that holds an infinity or NaN
constexpr int OZ_ZERO = INT_MIN / 2;          // of a row of zeros

// one operand as rows (of op(A), or columns of op(B)) by K: entry (i, k) at p[i si + k sk]
struct OzOperand {
  const double2* p;
  long si, sk, sb;      // strides of a row, of k, of a batch entry
  int rows, conj, kneg; // kneg: +1 scales by 2^g_k (A), -1 by 2^-g_k (B)
  const double* dk;     // optional diagonal along K
  __nv_bfloat16* out;   // planes [batch][slice][row'][k']
  int* ex;              // row exponents [batch][rows]
  long plane;           // elements of one slice plane
};

// the entry with its diagonal factor and conjugation applied
__device__ __forceinline__ double2 oz_entry(const OzOperand& o, const double2* p, int i, int k) {
  double2 v = p[i * o.si + k * o.sk];
  if (o.dk) {
    const double s = o.dk[k];
    v.x *= s;
    v.y *= s;
  }
  if (o.conj) v.y = -v.y;
  return v;
}

__device__ __forceinline__ bool oz_zero(double2 v) {  // without the FP64 pipe
  return !(((__double2hiint(v.x) | __double2hiint(v.y)) & 0x7fffffff) | __double2loint(v.x) | __double2loint(v.y));
}

// Biased exponent of x (subnormals: 1), OZ_ZERO for 0; 0x7ff for infinities and NaN.  One more when
// the fraction is within 2^-7 of the next binade, so that |x| < 0.9922 * 2^(e - 1022): seven signed
// bytes, -128 .. 127, reach 127/255 of 256^7, 0.9961 of 2^55.
__device__ __forceinline__ int oz_exp(double x) {
  const int hi = __double2hiint(x) & 0x7fffffff;
  if (!(hi | __double2loint(x))) return OZ_ZERO;
  if (hi >= 0x7ff00000) return 0x7ff;
  return min(max((hi + 0x4000) >> 20, 1), 0x7fe);
}

// g[k] = (exponent of the largest component in row k of op(B)) - 1023; 0 for rows of zeros and for
// rows with non-finite entries.  4 k's and 64 lanes along the row per CTA: 64-byte segments when k is
// contiguous, and enough CTAs at K = 256 (32 k's per CTA left 19 us on 8 CTAs there; now 4).
constexpr int KMAX_K = 4;
__global__ void __launch_bounds__(256) oz_kmax_k(const OzOperand b, int K, int* __restrict__ g) {
  __shared__ int red[8][KMAX_K];
  const int z = blockIdx.z, tid = threadIdx.x;
  const double2* p = b.p + z * b.sb;
  const int kk = tid % KMAX_K, k = blockIdx.x * KMAX_K + kk;
  int e = OZ_ZERO;
  if (k < K) {
#pragma unroll 4
    for (int j = tid / KMAX_K; j < b.rows; j += 256 / KMAX_K) {
      const double2 v = p[j * b.si + k * b.sk];
      e = max(e, max(oz_exp(v.x), oz_exp(v.y)));
    }
  }
  for (int o = 16; o >= KMAX_K; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if ((tid & 31) < KMAX_K) red[tid >> 5][kk] = e;
  __syncthreads();
  if (tid < KMAX_K && k < K) {
    for (int w = 1; w < 8; w++) e = max(e, red[w][kk]);
    g[(long)z * K + k] = (e == OZ_ZERO || e == 0x7ff) ? 0 : e - 1023;
  }
}

// 56-bit fixed point (sign included) of x 2^g relative to the row exponent E (|x| < 0.9922 2^(E - 1022)),
// rounded, plus the byte bias that turns its base-256 digits into q + 128
__device__ __forceinline__ unsigned long long oz_fixed(double x, int shift) {
  const unsigned long long kBias = 0x80808080808080ull;
  const long long bits = __double_as_longlong(x);
  const int e = (int)((bits >> 52) & 0x7ff);
  unsigned long long m = (unsigned long long)bits & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int sh = shift - max(e, 1);  // right shift; -2 for the leading binade
  unsigned long long v;
  if (sh <= 0) v = m << min(-sh, 2);
  else if (sh > 54) v = 0;
  else v = (m + (1ull << (sh - 1))) >> sh;
  return bits < 0 ? kBias - v : kBias + v;
}
// slice s of four biased values as four bf16, times `scale` (a power of two)
__device__ __forceinline__ uint2 oz_slice4(const unsigned long long (&v)[4], int s, float scale) {
  float f[4];
#pragma unroll
  for (int u = 0; u < 4; u++)
    f[u] = (__uint_as_float(0x4B000000u | (unsigned)((v[u] >> (8 * (OZ_S - 1 - s))) & 0xff)) - 8388736.f) * scale;
  const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
  return make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}

// the weight of slice s (accumulator d) with the guard, 2^(-8 s), and its inverse
__device__ __forceinline__ float oz_down(int s) { return __uint_as_float((unsigned)(127 - 8 * s) << 23); }
__device__ __forceinline__ float oz_up(int d) { return __uint_as_float((unsigned)(127 + 8 * d) << 23); }

// RB rows of one operand per CTA: exponents, then digits through a shared tile of 1024 / RB k's.
template <int RB>
__global__ void __launch_bounds__(256) oz_digits_k(const OzOperand a, const OzOperand b, int K, int Kh,
                                                   const int* __restrict__ g, long gstride, int nba, int nbb, int batch,
                                                   int planes) {
  constexpr int KC = 1024 / RB, KL = 256 / RB;
  __shared__ double2 tile[RB][KC + 1];
  __shared__ int emax[RB];
  const int tid = threadIdx.x;
  const bool is_a = (int)blockIdx.x < nba * batch;
  const OzOperand& o = is_a ? a : b;
  const int blk = is_a ? blockIdx.x : blockIdx.x - nba * batch;
  const int per = is_a ? nba : nbb, z = blk / per, i0 = (blk % per) * RB;
  const double2* p = o.p + z * o.sb;
  g += z * gstride;
  // row fastest when rows are contiguous in memory, else k fastest
  const bool rfast = o.si == 1;
  const int lr = rfast ? tid % RB : tid / KL, lk = rfast ? tid / RB : tid % KL;
  if (tid < RB) emax[tid] = OZ_ZERO;
  __syncthreads();
  if (i0 + lr < o.rows) {
    int e = OZ_ZERO;
#pragma unroll 4
    for (int k = lk; k < K; k += KL) {
      const double2 v = oz_entry(o, p, i0 + lr, k);
      const int ev = max(oz_exp(v.x), oz_exp(v.y));
      if (ev == 0x7ff) e = INT_MAX;
      else if (ev != OZ_ZERO) e = max(e, ev + o.kneg * g[k]);
    }
    atomicMax(&emax[lr], e);
  }
  __syncthreads();
  if (tid < RB && i0 + tid < o.rows) o.ex[(long)z * o.rows + i0 + tid] = emax[tid] == INT_MAX ? OZ_BAD : emax[tid];
  const int r = tid / (KC / 4), k4 = (tid % (KC / 4)) * 4;
  const int i = i0 + r, E = min(emax[r], 1 << 20);
  const long Kp = 2L * Kh;
  __nv_bfloat16* out = o.out + (long)z * planes * o.plane;
  for (int k0 = 0; k0 < Kh; k0 += KC) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int k = k0 + lk + q * KL;
      double2 v = make_double2(0.0, 0.0);
      if (i0 + lr < o.rows && k < K) v = oz_entry(o, p, i0 + lr, k);
      tile[lr][lk + q * KL] = v;
    }
    __syncthreads();
    const int k = k0 + k4;
    if (i >= o.rows || k >= Kh) continue;
    unsigned long long vr[4], vi[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const double2 v = tile[r][k4 + u];
      const int sh = E - 2 - (k + u < K ? o.kneg * g[k + u] : 0);
      vr[u] = oz_fixed(v.x, sh);
      vi[u] = oz_fixed(v.y, sh);
    }
#pragma unroll
    for (int s = 0; s <= OZ_S; s++) {
      if (s == OZ_S && planes == OZ_S) break;
      const float scale = planes == OZ_S ? 1.f : oz_down(s % OZ_S);
      uint2 re = oz_slice4(vr, s % OZ_S, scale), im = oz_slice4(vi, s % OZ_S, scale);
      if (s == OZ_S) {  // the guard's plane
        re = make_uint2(re.x & 0x7fff7fffu, re.y & 0x7fff7fffu);
        im = make_uint2(im.x & 0x7fff7fffu, im.y & 0x7fff7fffu);
      }
      __nv_bfloat16* pl = out + s * o.plane;
      if (is_a) {
        const uint2 ng = s == OZ_S ? im : make_uint2(im.x ^ 0x80008000u, im.y ^ 0x80008000u);
        const long rre = (long)(i / 64) * 128 + (i % 64), rim = rre + 64;
        *reinterpret_cast<uint2*>(pl + rre * Kp + k) = re;
        *reinterpret_cast<uint2*>(pl + rre * Kp + Kh + k) = ng;
        *reinterpret_cast<uint2*>(pl + rim * Kp + k) = im;
        *reinterpret_cast<uint2*>(pl + rim * Kp + Kh + k) = re;
      } else {
        *reinterpret_cast<uint2*>(pl + (long)i * Kp + k) = re;
        *reinterpret_cast<uint2*>(pl + (long)i * Kp + Kh + k) = im;
      }
    }
  }
}

// Shared-memory descriptor of a K-major tile with 64-byte rows and the 64-byte swizzle (layout type 4,
// 512 B between 8-row groups).
__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)4 << 61);
}
constexpr uint32_t kOzIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_BN >> 3) << 17) |
                              ((uint32_t)(OZ_BM >> 4) << 24);
// The descriptors of a stage's tiles differ in their low words only.
__device__ __forceinline__ void oz_mma(uint32_t d, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}" ::"r"(d),
      "r"(alo), "r"(blo), "r"(hi), "r"(kOzIdesc), "r"(accumulate)
      : "memory");
}
// the products of accumulators D0 <= d < D1 of one stage; with the guard those of d = 7 go into the last one
template <int D0, int D1, bool GUARD>
__device__ __forceinline__ void oz_products(uint32_t tmem, uint32_t alo, uint32_t blo, uint32_t hi, bool first) {
#pragma unroll
  for (int d = D0; d < D1; d++)
#pragma unroll
    for (int i = 0; i <= d; i++)
#pragma unroll
      for (int j = 0; j < OZ_BK / 16; j++)
        oz_mma(tmem + (uint32_t)(d * OZ_BN), alo + (uint32_t)((i * OZ_AT + 32 * j) >> 4),
               blo + (uint32_t)(((d - i) * OZ_BT + 32 * j) >> 4), hi, (first && i == 0 && j == 0) ? 0u : 1u);
  if (GUARD && D1 == OZ_S) {
#pragma unroll
    for (int i = 1; i < OZ_S; i++)
#pragma unroll
      for (int j = 0; j < OZ_BK / 16; j++)
        oz_mma(tmem + (uint32_t)((OZ_S - 1) * OZ_BN), alo + (uint32_t)((i * OZ_AT + 32 * j) >> 4),
               blo + (uint32_t)(((OZ_S - i) * OZ_BT + 32 * j) >> 4), hi, 1u);
  }
}
__device__ __forceinline__ void oz_tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
// acc += w * (16 accumulator columns, times `up`, as integers).  Sums below 2^22 (nearly always) turn into integers
// by adding 1.5 2^23 and reading the bits; the conversion instruction runs at an eighth of that rate.
template <bool GUARD>
__device__ __forceinline__ void oz_drain(uint32_t ta, int w, float up, long long (&acc)[16]) {
  float v[16];
  oz_tmem_ld16(ta, v);
  if (GUARD) {
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] *= up;
  }
  float top = 0.f;
#pragma unroll
  for (int j = 0; j < 16; j++) top = fmaxf(top, fabsf(v[j]));
  if (__all_sync(0xffffffffu, top < 4194304.f)) {
#pragma unroll
    for (int j = 0; j < 16; j++) acc[j] += (long long)(__float_as_int(v[j] + 12582912.f) - 0x4B400000) * w;
  } else {
#pragma unroll
    for (int j = 0; j < 16; j++) acc[j] += (long long)__float2int_rn(v[j]) * w;
  }
}
__device__ __forceinline__ void oz_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t oz_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float oz_ldf_remote(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ longlong2 oz_ld_remote(uint32_t addr) {
  longlong2 v;
  asm volatile("ld.shared::cluster.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr) : "memory");
  return v;
}
// (hi 2^32 + lo) 2^e in FP64: one rounding of the integer, then an exact scaling
__device__ __forceinline__ double oz_double(long long hi, long long lo, int e) {
  hi += lo >> 32;
  const unsigned l = (unsigned)lo;
  if (!(hi | (long long)l)) return 0.0;
  // 1.5 2^52 + hi and 2^20 + l 2^-32 as bit patterns; the two offsets leave in the first subtraction
  const double dh = __longlong_as_double(0x4338000000000000ll + hi) - (6755399441055744.0 + 1048576.0);
  const double r = dh + __longlong_as_double(0x4130000000000000ll | (long long)l);
  const long long rb = __double_as_longlong(r);
  const int ne = (int)((rb >> 52) & 0x7ff) + e;
  if (ne > 0 && ne < 0x7ff) return __longlong_as_double(rb + ((long long)e << 52));
  return scalbn(scalbn(r, e / 2), e - e / 2);
}

// The least sum of the guard's products per sqrt(K).  Gaussian entries give ~1000 K; rows with one entry that
// counts (a diagonal environment) ~127 times the other operand's leading byte.
constexpr float OZ_LEAST = 16.f;
// what the epilogue needs to form an element in plain FP64
struct OzPlain {
  OzOperand a, b;
  int K;
};

template <bool GUARD>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    zgemm_oz_k(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, double2* __restrict__ C,
               long ldc, long sC, int M, int N, int nk, int bshared, int ntm, int ntn, int cs, int herm,
               int sub, float least, const OzPlain plain) {
  constexpr int NP = oz_planes(GUARD), OZ_STAGE = oz_stage(GUARD);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OZ_STAGES * OZ_STAGE);
  uint64_t* full = bars;                    // [stages] loaded
  uint64_t* empty = bars + OZ_STAGES;       // [stages] consumed by the MMAs
  uint64_t* afull = bars + 2 * OZ_STAGES;   // [H, L] accumulators hold a chunk
  uint64_t* aempty = afull + 2;             // [H, L] accumulators drained
  uint64_t* done = afull + 4;               // all MMAs complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(afull + 5);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(afull + 6);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x % cs;
  int t = blockIdx.x / cs, tn = t % ntn, tm = (t / ntn) % ntm, z = t / (ntn * ntm);
  if (herm) {  // the tiles on and above the diagonal, by columns of tiles: t = tn (tn + 1) / 2 + tm
    tn = (int)((sqrtf(8.f * t + 1.f) - 1.f) * 0.5f);
    while (tn * (tn + 1) / 2 > t) tn--;
    while ((tn + 1) * (tn + 2) / 2 <= t) tn++;
    tm = t - tn * (tn + 1) / 2;
    z = 0;
  }
  const int kb0 = (int)((long)nk * rank / cs), kb1 = (int)((long)nk * (rank + 1) / cs);

  if (threadIdx.x == 0) {
    for (int s = 0; s < OZ_STAGES; s++) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(afull + i, 1);
      mbar_init(aempty + i, OZ_EPI_WARPS);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(OZ_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  longlong2* sums = reinterpret_cast<longlong2*>(smem);  // [column][row] (hi, lo), once the stages are free
  float* gsums = reinterpret_cast<float*>(smem + OZ_SUMS);                       // [column][row], with the guard
  unsigned* nlist = reinterpret_cast<unsigned*>(smem + OZ_SUMS + OZ_GSUMS);      // elements to form in FP64
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + OZ_SUMS + OZ_GSUMS + 16);

  if (warp == 0) {
    if (elect_one()) {
      const int arow = tm * OZ_BM, brow = tn * OZ_BN, apl = NP * z, bpl = bshared ? 0 : NP * z;
      int issued[OZ_STAGES] = {0, 0};
      bool ok = true;
      for (int kb = kb0; kb < kb1; kb++) {
        const int n = kb - kb0, s = n % OZ_STAGES;
        if (*abort_flag || !mbar_wait(empty + s, ((n / OZ_STAGES) & 1u) ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        uint8_t* st = smem + s * OZ_STAGE;
        mbar_expect_tx(full + s, OZ_STAGE);
        for (int sl = 0; sl < NP; sl++) {
          tma_load_3d(st + sl * OZ_AT, &tmA, kb * OZ_BK, arow, apl + sl, full + s);
          tma_load_3d(st + NP * OZ_AT + sl * OZ_BT, &tmB, kb * OZ_BK, brow, bpl + sl, full + s);
        }
        issued[s]++;
      }
      if (!ok) *abort_flag = 1;
      // every copy this thread started has landed before the CTA may exit
      for (int s = 0; s < OZ_STAGES; s++)
        if (issued[s] > 0 && !mbar_wait(full + s, (uint32_t)(issued[s] - 1) & 1u, &kNever)) *abort_flag = 1;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = true;
      const int last = kb1 - kb0 - 1;
      unsigned chunk[2] = {0, 0};
      bool first[2] = {true, true};  // the group's accumulators start from zero
      for (int n = 0; n <= last && ok; n++) {
        const int s = n % OZ_STAGES;
        if (*abort_flag || !mbar_wait(full + s, (n / OZ_STAGES) & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint64_t da = oz_desc(smem_u32(smem + s * OZ_STAGE)), db = oz_desc(smem_u32(smem + s * OZ_STAGE) + NP * OZ_AT);
        const uint32_t dh = (uint32_t)(da >> 32);
        if (GUARD) {  // into the columns behind the seven accumulators, drained once, with the last chunks
#pragma unroll
          for (int j = 0; j < OZ_BK / 16; j++)
            oz_mma(tmem + OZ_S * OZ_BN, (uint32_t)da + (uint32_t)((OZ_S * OZ_AT + 32 * j) >> 4),
                   (uint32_t)db + (uint32_t)((OZ_S * OZ_BT + 32 * j) >> 4), dh, n > 0 || j > 0 ? 1u : 0u);
        }
        // the group that is being drained comes second
        for (int o = 0; o < 2; o++) {
          const bool low = first[1] ? o == 1 : o == 0;
          const int grp = low ? 1 : 0;
          if (first[grp]) {
            if (*abort_flag || !mbar_wait(aempty + grp, (chunk[grp] & 1u) ^ 1u, abort_flag)) { ok = false; break; }
            tc_fence_after();
          }
          const bool f = first[grp];
          first[grp] = false;
          if (low) oz_products<OZ_DH, OZ_S, GUARD>(tmem, (uint32_t)da, (uint32_t)db, dh, f);
          else oz_products<0, OZ_DH, GUARD>(tmem, (uint32_t)da, (uint32_t)db, dh, f);
        }
        if (!ok) break;
        tc_commit(empty + s);
        if (oz_drain_h(n, last)) {
          tc_commit(afull);
          chunk[0]++;
          first[0] = true;
        }
        if (oz_drain_l(n, last)) {
          tc_commit(afull + 1);
          chunk[1]++;
          first[1] = true;
        }
      }
      if (!ok) *abort_flag = 1;
      tc_commit(done);
      if (!mbar_wait(done, 0, &kNever)) *abort_flag = 1;
    }
    __syncwarp();
  } else {
    // warp w drains TMEM lanes 32 (w % 4) .. + 31 and OZ_EC of the 64 columns
    constexpr int OZ_EC = OZ_BN * 4 / OZ_EPI_WARPS;
    static_assert(OZ_EC == 16, "oz_drain reads 16 columns");
    const int q = warp & 3, part = (warp - 2) >> 2;
    long long hi[OZ_EC], lo[OZ_EC];
#pragma unroll
    for (int j = 0; j < OZ_EC; j++) hi[j] = lo[j] = 0;
    bool ok = true;
    const int last = kb1 - kb0 - 1;
    unsigned chunk[2] = {0, 0};
    const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(part * OZ_EC);
    // one group of accumulators complete: lane 0 waits and the warp follows its verdict
    auto wait_group = [&](int grp) {
      int got = 0;
      if (lane == 0) got = (!*abort_flag && mbar_wait(afull + grp, chunk[grp] & 1u, abort_flag)) ? 1 : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      chunk[grp]++;
      tc_fence_after();
      return got != 0;
    };
    auto release = [&](int grp) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(aempty + grp);
    };
    for (int n = 3; ok; n += 4) {
      n = min(n, last);
      if (oz_drain_h(n, last)) {
        if (!(ok = wait_group(0))) break;
        int w = 1 << 16;
#pragma unroll 1
        for (int d = 0; d < 3; d++, w >>= 8) oz_drain<GUARD>(ta + d * OZ_BN, w, oz_up(d), hi);
        oz_drain<GUARD>(ta + 3 * OZ_BN, 1 << 24, oz_up(3), lo);
        release(0);
      }
      if (oz_drain_l(n, last)) {
        if (!(ok = wait_group(1))) break;
        int w = 1 << 16;
#pragma unroll 1
        for (int d = OZ_DH; d < OZ_S; d++, w >>= 8) oz_drain<GUARD>(ta + d * OZ_BN, w, oz_up(d), lo);
        release(1);
      }
      if (n == last) break;
    }
    if (!ok) *abort_flag = 1;
    // after the last chunk the stages are free: every MMA has read them
    if (ok) {
      longlong2* o = sums + (long)(part * OZ_EC) * OZ_BM + 32 * q + lane;
#pragma unroll
      for (int j = 0; j < OZ_EC; j++) o[j * OZ_BM] = make_longlong2(hi[j], lo[j]);
      if (GUARD) {
        float v[16];
        oz_tmem_ld16(ta + OZ_S * OZ_BN, v);
        float* p = gsums + (part * OZ_EC) * OZ_BM + 32 * q + lane;
#pragma unroll
        for (int j = 0; j < OZ_EC; j++) p[j * OZ_BM] = v[j];
        if (warp == 2 && lane == 0) *nlist = 0;
      }
    }
  }
  tc_fence_before();
  if (cs > 1) oz_cluster_sync();
  else __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_TMEM_COLS) : "memory");
  // this CTA rounds and stores 64 / cs of the tile's columns
  const uint32_t sbase = smem_u32(sums), gbase = smem_u32(gsums), fbase = smem_u32(const_cast<const uint32_t*>(abort_flag));
  bool bad = false;
  for (int r = 0; r < cs; r++) {
    uint32_t f;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(f) : "r"(oz_map(fbase, r)) : "memory");
    bad = bad || f;
  }
  const int nc = OZ_BN / cs;
  const int* ea = plain.a.ex + (long)z * M;
  const int* eb = plain.b.ex + (bshared ? 0 : (long)z * N);
  for (int e = threadIdx.x; e < 64 * nc; e += OZ_THREADS) {
    const int i = e & 63, c = rank * nc + (e >> 6);
    const int gi = tm * 64 + i, gj = tn * OZ_BN + c;
    if (gi >= M || gj >= N || (herm && gi > gj)) continue;
    double2 out;
    const int xa = ea[gi], xb = eb[gj];
    if (bad) {
      out.x = out.y = __longlong_as_double(0x7ff8000000000000ll);  // a bounded wait gave up
    } else if (xa == OZ_BAD || xb == OZ_BAD) {
      const double2 *pa = plain.a.p + z * plain.a.sb, *pb = plain.b.p + (bshared ? 0 : z * plain.b.sb);
      out = make_double2(0.0, 0.0);
      for (int k = 0; k < plain.K; k++) out = cadd(out, cmul(oz_entry(plain.a, pa, gi, k), oz_entry(plain.b, pb, gj, k)));
      out = cmul(make_double2(1.0, 0.0), out);  // alpha of the general product: 0 x infinity is NaN
    } else if (xa == OZ_ZERO || xb == OZ_ZERO) {
      out.x = out.y = 0.0;
    } else {
      longlong2 re = make_longlong2(0, 0), im = re;
      float p = 0.f;
      for (int r0 = 0; r0 < cs; r0 += 2) {  // cs is 1 or even: two ranks' loads in flight
        longlong2 x[2], y[2];
        float px[2] = {0.f, 0.f}, py[2] = {0.f, 0.f};
#pragma unroll
        for (int u = 0; u < 2; u++)
          if (r0 + u < cs) {
            const uint32_t at = oz_map(sbase + (uint32_t)(c * OZ_BM + i) * 16u, r0 + u);
            x[u] = oz_ld_remote(at);
            y[u] = oz_ld_remote(at + 64 * 16);
            if (GUARD) {
              const uint32_t gat = oz_map(gbase + (uint32_t)(c * OZ_BM + i) * 4u, r0 + u);
              px[u] = oz_ldf_remote(gat);
              py[u] = oz_ldf_remote(gat + 64 * 4);
            }
          } else {
            x[u] = y[u] = make_longlong2(0, 0);
          }
        re.x += x[0].x + x[1].x;
        re.y += x[0].y + x[1].y;
        im.x += y[0].x + y[1].x;
        im.y += y[0].y + y[1].y;
        if (GUARD) p += (px[0] + py[0]) + (px[1] + py[1]);
      }
      if (GUARD && p < least) {
        list[atomicAdd(nlist, 1u)] = (uint16_t)e;
        continue;
      }
      // units: q q' of slices 6 is 2^(E_i - 1077 + E_j - 1077); the sums carry 2^48 and hi 2^32 of it
      const int sc = xa + xb - 2154 + 48 + 32;
      out.x = oz_double(re.x, re.y, sc);
      out.y = oz_double(im.x, im.y, sc);
    }
    if (sub) out = csub(C[z * sC + gi + (long)gj * ldc], out);
    C[z * sC + gi + (long)gj * ldc] = out;
    if (herm && gi != gj) C[gj + (long)gi * ldc] = cconj(out);
  }
  __syncwarp();
  if (cs > 1) oz_cluster_sync();  // the sums stay readable until every CTA of the cluster has them
  else if (GUARD) __syncthreads();
  if (GUARD && !bad) {  // a warp an element, lanes along K
    const int n = (int)*nlist;
    for (int f = warp; f < n; f += OZ_THREADS / 32) {
      const int e = list[f], gi = tm * 64 + (e & 63), gj = tn * OZ_BN + rank * nc + (e >> 6);
      const double2 *pa = plain.a.p + z * plain.a.sb, *pb = plain.b.p + (bshared ? 0 : z * plain.b.sb);
      double2 out = make_double2(0.0, 0.0);
      for (int k = lane; k < plain.K; k += 32) {
        // (zeros, of which such operands are often full, cost the FP64 pipe nothing; the other factor is finite here)
        if (oz_zero(pa[gi * plain.a.si + k * plain.a.sk]) || oz_zero(pb[gj * plain.b.si + k * plain.b.sk])) continue;
        const double2 x = oz_entry(plain.a, pa, gi, k), y = oz_entry(plain.b, pb, gj, k);
        out.x = fma(x.x, y.x, fma(-x.y, y.y, out.x));
        out.y = fma(x.x, y.y, fma(x.y, y.x, out.y));
      }
      __syncwarp();
      for (int o = 16; o > 0; o >>= 1) {
        out.x += __shfl_xor_sync(0xffffffffu, out.x, o);
        out.y += __shfl_xor_sync(0xffffffffu, out.y, o);
      }
      if (lane != 0) continue;
      if (sub) out = csub(C[z * sC + gi + (long)gj * ldc], out);
      C[z * sC + gi + (long)gj * ldc] = out;
      if (herm && gi != gj) C[gj + (long)gi * ldc] = cconj(out);
    }
  }
}

int oz_map_make(CUtensorMap* map, const void* base, long Kp, long rows, long planes, int box_rows) {
  EncodeTiled enc = nullptr;
  QR_TRY(encode_fn(&enc));
  cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
  cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(Kp * 2 * rows)};
  cuuint32_t box[3] = {OZ_BK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(QR_ECUDA, "cuTensorMapEncodeTiled failed (code " + std::to_string((int)r) + ")");
  return QR_OK;
}

// clusters of `cs` CTAs the device holds at once
int oz_clusters(bool guard, int cs, int* out) {
  static std::mutex mu;
  static std::map<std::tuple<int, bool, int>, int> known;
  int dev = 0;
  QR_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto it = known.find({dev, guard, cs});
  if (it == known.end()) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(OZ_THREADS);
    cfg.dynamicSmemBytes = oz_smem(guard);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (guard) QR_CUDA(cudaOccupancyMaxActiveClusters(&n, zgemm_oz_k<true>, &cfg));
    else QR_CUDA(cudaOccupancyMaxActiveClusters(&n, zgemm_oz_k<false>, &cfg));
    it = known.emplace(std::make_tuple(dev, guard, cs), n).first;
  }
  *out = it->second;
  return QR_OK;
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

// Largest K of the integer sums (hi stays below 2^51) and the largest plane rows TMA addresses.
bool zgemm_oz_fits(int M, int N, int K) { return K <= (1 << 20) && M <= (1 << 28) && N <= (1 << 28); }

// Workspace for slices at a time: a batch that needs more goes through in runs of whole entries.
constexpr size_t OZ_ROOM = (size_t)1 << 30;
constexpr int OZ_NO_ROOM = -1;  // oz_run: the slices found no memory, nothing was launched

static int oz_run(cudaStream_t s, int opA, int opB, int M, int N, int K, const double2* A, long lda, long sA,
                  const double2* B, long ldb, long sB, double2* C, long ldc, long sC, int batch, const double* dk,
                  int herm, int eq_a, int sub, bool guard, size_t room = OZ_ROOM) {
  if (room == 0) return OZ_NO_ROOM;
  const int planes = oz_planes(guard);
  const float least = OZ_LEAST * sqrtf((float)K);
  const bool bshared = sB == 0 || batch == 1;
  const int ntm = (M + 63) / 64, ntn = (N + OZ_BN - 1) / OZ_BN, Kh = (K + 15) / 16 * 16;
  const long Kp = 2L * Kh, arows = 128L * ntm, brows = (long)OZ_BN * ntn;
  const long apl = arows * Kp, bpl = brows * Kp;
  // bytes of one entry of A, and of B with its scales along K
  const size_t abytes = (size_t)planes * apl * 2 + sizeof(int) * (size_t)M;
  const size_t bbytes = (size_t)planes * bpl * 2 + sizeof(int) * ((size_t)N + K);
  const size_t fixed = bshared ? bbytes : 0, each = abytes + (bshared ? 0 : bbytes);
  int run_len = (int)std::min<size_t>(batch, std::max<size_t>(1, room > fixed ? (room - fixed) / each : 1));
  char* ws = nullptr;
  int bb = 1;
  size_t ab = 0, bbt = 0, ea = 0, eb = 0;
  for (;;) {
    bb = bshared ? 1 : run_len;
    ab = up256((size_t)run_len * planes * apl * 2);
    bbt = up256((size_t)bb * planes * bpl * 2);
    ea = up256(sizeof(int) * (size_t)run_len * M);
    eb = up256(sizeof(int) * (size_t)bb * N);
    const cudaError_t e = cudaMallocAsync((void**)&ws, ab + bbt + ea + eb + sizeof(int) * (size_t)bb * K, s);
    if (e == cudaSuccess) break;
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "GEMM slices");
    (void)cudaGetLastError();  // not an error of the next launch
    if (run_len == 1) return OZ_NO_ROOM;
    run_len = (run_len + 1) / 2;
  }
  int* g = (int*)(ws + ab + bbt + ea + eb);
  const bool an = opA == OP_N || opA == OP_R, bn = opB == OP_N || opB == OP_R;
  // entries z0 .. z0 + nz - 1
  auto run = [&](int z0, int nz) -> int {
    const int nb = bshared ? 1 : nz;
    const bool slice_b = !bshared || z0 == 0;
    OzPlain pl;
    pl.K = K;
    pl.a = {A + z0 * sA, an ? 1 : lda, an ? lda : 1, sA, M, opA == OP_C || opA == OP_R, eq_a ? -1 : 1, dk,
            (__nv_bfloat16*)ws, (int*)(ws + ab + bbt), apl};
    pl.b = {bshared ? B : B + z0 * sB, bn ? ldb : 1, bn ? 1 : ldb, bshared ? 0 : sB, N, opB == OP_C || opB == OP_R,
            eq_a ? 1 : -1, nullptr, (__nv_bfloat16*)(ws + ab), (int*)(ws + ab + bbt + ea), bpl};
    if (slice_b) {
      oz_kmax_k<<<dim3(ceil_div(K, KMAX_K), 1, nb), 256, 0, s>>>(eq_a ? pl.a : pl.b, K, g);
      QR_CHECK_LAUNCH("oz_kmax_k");
    }
    // up to 16 rows for each of the 152 SMs: 4 per CTA so that the pass still covers them; else 16
    const long rows = (long)M * nz + (slice_b ? (long)N * nb : 0);
    const int rb = rows <= 2432 ? 4 : 16;
    const int nba = (M + rb - 1) / rb, nbb = (N + rb - 1) / rb;
    const unsigned grid = (unsigned)((long)nba * nz + (slice_b ? (long)nbb * nb : 0));
    const long gs = bshared ? 0 : K;
    if (rb == 4) oz_digits_k<4><<<grid, 256, 0, s>>>(pl.a, pl.b, K, Kh, g, gs, nba, nbb, nz, planes);
    else oz_digits_k<16><<<grid, 256, 0, s>>>(pl.a, pl.b, K, Kh, g, gs, nba, nbb, nz, planes);
    QR_CHECK_LAUNCH("oz_digits_k");
    CUtensorMap ma, mb;
    QR_TRY(oz_map_make(&ma, ws, Kp, arows, (long)planes * nz, OZ_BM));
    QR_TRY(oz_map_make(&mb, ws + ab, Kp, brows, (long)planes * nb, OZ_BN));
    auto kern = guard ? zgemm_oz_k<true> : zgemm_oz_k<false>;
    QR_TRY(set_func_attr_once((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, oz_smem(guard)));
    const int nk = (int)(Kp / OZ_BK);
    const long tiles = herm ? (long)ntm * (ntm + 1) / 2 : (long)ntm * ntn * nz;
    // K split over a cluster: the split with the fewest (waves x stages per CTA), a CTA's fixed cost
    // counted as 5 stages and a split's as 2 more
    int cs = 1;
    double best = 1e300;
    for (int c = 1; c <= 8 && c <= nk; c *= 2) {
      int resident = 0;
      QR_TRY(oz_clusters(guard, c, &resident));
      if (resident < 1) continue;
      const double cost = (double)ceil_div(tiles, resident) * (ceil_div(nk, c) + 5.0 + (c > 1 ? 2.0 : 0.0));
      if (cost < best) {
        best = cost;
        cs = c;
      }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * cs));
    cfg.blockDim = dim3(OZ_THREADS);
    cfg.dynamicSmemBytes = oz_smem(guard);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    QR_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mb, C + z0 * sC, ldc, sC, M, N, nk, bshared ? 1 : 0, ntm, ntn, cs, herm,
                               sub, least, pl));
    count_launch();
    return QR_OK;
  };
  int rc = QR_OK;
  for (int z0 = 0; z0 < batch && !rc; z0 += run_len) rc = run(z0, std::min(run_len, batch - z0));
  cudaFreeAsync(ws, s);
  return rc;
}

// (where the slices find no memory, the products run on the CUDA cores, which need none)
int zgemm_oz(cudaStream_t s, int opA, int opB, int M, int N, int K, const double2* A, long lda, long sA,
             const double2* B, long ldb, long sB, double2* C, long ldc, long sC, int batch, const double* dk, bool guard,
             size_t room) {
  const int rc = oz_run(s, opA, opB, M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, dk, 0, 0, 0, guard, room);
  if (rc != OZ_NO_ROOM) return rc;
  return zgemm_spread(s, opA, opB, M, N, K, make_double2(1.0, 0.0), A, lda, sA, B, ldb, sB, make_double2(0.0, 0.0), C, ldc,
                      sC, batch, dk);
}
int zgemm_oz(cudaStream_t s, int opA, int opB, int M, int N, int K, const double2* A, long lda, long sA,
             const double2* B, long ldb, long sB, double2* C, long ldc, long sC, int batch, const double* dk, bool guard) {
  return zgemm_oz(s, opA, opB, M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, dk, guard, OZ_ROOM);
}

// C = A B (M x K, K x N) for an A whose columns spread over decades: the scaling along K equilibrates A's
// columns instead of B's rows, so columns of C that combine small columns of A keep their relative accuracy
int zgemm_graded(cudaStream_t s, int M, int N, int K, const double2* A, long lda, const double2* B, long ldb, double2* C,
                 long ldc) {
  const double work = (double)M * N * K;
  if (work < OZ_MIN_WORK || !zgemm_oz_fits(M, N, K))
    return zgemm(s, OP_N, OP_N, M, N, K, make_double2(1.0, 0.0), A, lda, 0, B, ldb, 0, make_double2(0.0, 0.0), C, ldc, 0,
                 1, nullptr);
  const int pr = prof_begin(s, PK_ZGEMM, 8.0 * work, 16.0 * ((double)M * K + (double)K * N + (double)M * N));
  int rc = oz_run(s, OP_N, OP_N, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, nullptr, 0, 1, 0, false);
  if (rc == OZ_NO_ROOM)
    rc = zgemm_spread(s, OP_N, OP_N, M, N, K, make_double2(1.0, 0.0), A, lda, 0, B, ldb, 0, make_double2(0.0, 0.0), C, ldc,
                      0, 1, nullptr);
  prof_end(s, pr);
  return rc;
}

// C -= A B (M x K, K x N)
int zgemm_sub(cudaStream_t s, int M, int N, int K, const double2* A, long lda, const double2* B, long ldb, double2* C,
              long ldc) {
  if (M <= 0 || N <= 0 || K <= 0) return QR_OK;
  const double work = (double)M * N * K;
  const int pr = prof_begin(s, PK_ZGEMM, 8.0 * work, 16.0 * ((double)M * K + (double)K * N + 2.0 * M * N));
  int rc = OZ_NO_ROOM;
  if (work >= OZ_MIN_WORK && zgemm_oz_fits(M, N, K))
    rc = oz_run(s, OP_N, OP_N, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, nullptr, 0, 0, 1, false);
  if (rc == OZ_NO_ROOM)
    rc = zgemm_spread(s, OP_N, OP_N, M, N, K, make_double2(-1.0, 0.0), A, lda, 0, B, ldb, 0, make_double2(1.0, 0.0), C, ldc,
                      0, 1, nullptr);
  prof_end(s, pr);
  return rc;
}

// C = A^H A (n x n, K rows): the entries on and above the diagonal, mirrored as they are stored (exactly
// Hermitian, which the rotations formed from a Gram matrix rely on)
int zherk(cudaStream_t s, int n, int K, const double2* A, long lda, double2* C, long ldc) {
  if (n <= 0) return QR_OK;
  const double work = (double)n * n * K;
  const int pr = prof_begin(s, PK_ZGEMM, 4.0 * work, 16.0 * ((double)n * K + (double)n * n));
  int rc = OZ_NO_ROOM;
  if (work >= OZ_MIN_WORK && zgemm_oz_fits(n, n, K))
    rc = oz_run(s, OP_C, OP_N, n, n, K, A, lda, 0, A, lda, 0, C, ldc, 0, 1, nullptr, 1, 0, 0, false);
  if (rc == OZ_NO_ROOM) rc = zherk_spread(s, n, K, A, lda, C, ldc);
  prof_end(s, pr);
  return rc;
}

}  // namespace qr
