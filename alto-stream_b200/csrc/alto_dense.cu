// Dense R x R and I x R kernels of CP-ALS and CP-stream, all in float64
// arithmetic over float32-stored factors.
//
// Reference operations (jeewhanchoi/ALTO-stream):
//   update_gram / mat_aTa (cblas_dsyrk)      src/gram.cpp:29-41, src/matrix.cpp:252-267
//   historical cross-Gram (cblas_dgemm)      src/streaming_cpd.cpp:1391-1400
//   hadamard_product / pseudo_inverse Hadamard src/matrix.cpp:269-294, include/cpd.hpp:383-397
//   Cholesky + solve (dpotrf/dpotrs)         include/cpd.hpp:409-476, src/matrix.cpp:226-250, 333-372
//   KruskalModelNorm                         src/kruskal_model.cpp:227-353
//   cpd_fit_alto                             include/cpd.hpp:193-275
//
// Reductions are deterministic: every kernel that reduces over rows writes
// per-block partials and a second kernel, or the last block to finish, sums
// them in block order.  The normal-equation solve forms the inverse of the Cholesky-
// factored R x R matrix once (one CTA) and applies it to all I rows as a
// float64 row-times-matrix product; the reference runs dpotrs over the rows.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "alto_dense.cuh"
#include "alto_dmma.cuh"
#include "alto_group.cuh"

namespace alto {

static int g_sms = 0;
static int sms() {
  if (!g_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 148;
  }
  return g_sms;
}

// ------------------------------------------------------------ Grams
//
// G = U^T U and, in the same pass, C = P^T U with the change statistics, as
// float64 tensor-core products over the rows.  A fragment of four rows by
// eight columns -- lane l holds (row l % 4, column l / 4), converted from the
// float32 element it loads -- is at once the A operand of the output tiles of
// its columns as rows and the B operand of those of its columns as columns, so
// a warp reads each element once, with no shared memory, and a step of four
// rows is T (T + 1) / 2 + T^2 products for 2 T loads (T = ceil(R / 8); G only
// on and above the diagonal tiles).  Bound by the float64 rate from rank 32
// (120,000 rows at rank 32: 12.5 us), by HBM below.  The form before staged the
// rows in shared memory and read two doubles for every multiply-add (61 us
// there; 109 us for 20,000 rows at rank 64, now 15).
//
// Up to rank 32 every warp of a block holds all tiles and takes its own rows;
// above, the block's eight warps share the rows and warp w holds the tiles of
// tile rows w, w + 8, ... (the accumulators of rank 64 are eight warps' registers).

constexpr int kGramThreads = 128;      // T <= 4
constexpr int kGramThreadsWide = 256;  // T > 4
constexpr int kGramBlocksPerSm = 2;

__host__ __device__ constexpr int gram_tiles(int R) { return (R + 7) / 8; }
// Output tiles, 64 doubles each, of one pass: G's on and above the diagonal,
// then C's.  Lane l of a tile's warp owns elements 2 l and 2 l + 1:
// (l / 4, 2 (l % 4)) and its right neighbour.
__host__ __device__ constexpr int gram_out_tiles(int T, bool cross) { return T * (T + 1) / 2 + (cross ? T * T : 0); }
__host__ __device__ constexpr int gram_tile_of(int T, int a, int b) { return a * T - a * (a - 1) / 2 + (b - a); }
// Doubles of one block's partial result (with the three statistics).
__host__ __device__ constexpr int gram_partial_len(int R, bool cross) {
  return gram_out_tiles(gram_tiles(R), cross) * 64 + (cross ? 3 : 0);
}

__device__ __forceinline__ void change_stats(double p, double u, double (&q)[3]) {
  const double d = p - u;
  q[0] = __fma_rn(p, u, q[0]);
  q[1] = __fma_rn(d, d, q[1]);
  q[2] = __fma_rn(u, u, q[2]);
}

// The block's three statistics: warp butterflies, then warps in order.
__device__ __forceinline__ void store_stats(double (&q)[3], double* __restrict__ out) {
  __shared__ double wq[3][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o; o >>= 1) q[k] += __shfl_xor_sync(0xffffffffu, q[k], o);
    if (lane == 0) wq[k][warp] = q[k];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += wq[threadIdx.x][w];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

// A Gram pass that first divides column c of U by lambda[c] (CP-ALS's
// normalisation): the scaled factor goes to Y, and in bfloat16 to shadow (may
// be NULL); U is left as it is.
struct GramScale {
  const double* lambda;
  float* Y;
  __nv_bfloat16* shadow;
};

// Partial sums over rows [r0, r1), T <= 4 column tiles.
template <int T, bool CROSS, bool SCALE>
__device__ __forceinline__ void gram_narrow(const float* __restrict__ P, const float* __restrict__ U, uint64_t r0,
                                            uint64_t r1, int R, double* __restrict__ out, const GramScale& sc) {
  constexpr int NG = T * (T + 1) / 2, NT = gram_out_tiles(T, CROSS), NW = kGramThreads / 32;
  constexpr int S = T == 1 ? 8 : T == 2 ? 4 : 2;  // steps of four rows whose loads are issued together
  __shared__ double red[NT * 64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kr = lane & 3, kc = lane >> 2;
  double acc[NT][2];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
  double q[3] = {0.0, 0.0, 0.0};
  double inv[SCALE ? T : 1];
  if constexpr (SCALE)
#pragma unroll
    for (int c = 0; c < T; ++c) inv[c] = c * 8 + kc < R ? 1.0 / sc.lambda[c * 8 + kc] : 0.0;
  float fu[S][T], fp[CROSS ? S : 1][T];
  auto fetch = [&](uint64_t k0) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const uint64_t row = k0 + (uint64_t)s * 4 * NW + kr;
#pragma unroll
      for (int c = 0; c < T; ++c) {
        const int col = c * 8 + kc;
        const bool ok = row < r1 && col < R;
        fu[s][c] = ok ? U[row * R + col] : 0.f;
        if (CROSS) fp[s][c] = ok ? P[row * R + col] : 0.f;
      }
    }
  };
  const uint64_t first = r0 + warp * 4;
  if (first < r1) fetch(first);
  for (uint64_t k0 = first; k0 < r1; k0 += (uint64_t)S * 4 * NW) {
    float cu[S][T], cp[CROSS ? S : 1][T];
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int c = 0; c < T; ++c) {
        cu[s][c] = fu[s][c];
        if (CROSS) cp[s][c] = fp[s][c];
      }
    if (k0 + (uint64_t)S * 4 * NW < r1) fetch(k0 + (uint64_t)S * 4 * NW);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      double u[T], p[T];
#pragma unroll
      for (int c = 0; c < T; ++c) {
        if constexpr (SCALE) {
          cu[s][c] = (float)((double)cu[s][c] * inv[c]);
          const uint64_t row = k0 + (uint64_t)s * 4 * NW + kr;
          const int col = c * 8 + kc;
          if (row < r1 && col < R) {
            sc.Y[row * R + col] = cu[s][c];
            if (sc.shadow) sc.shadow[row * R + col] = __float2bfloat16(cu[s][c]);
          }
        }
        u[c] = (double)cu[s][c];
        if (CROSS) {
          p[c] = (double)cp[s][c];
          change_stats(p[c], u[c], q);
        }
      }
#pragma unroll
      for (int a = 0; a < T; ++a)
#pragma unroll
        for (int b = a; b < T; ++b) dmma_8x8x4(acc[gram_tile_of(T, a, b)], u[a], u[b]);
      if (CROSS)
#pragma unroll
        for (int a = 0; a < T; ++a)
#pragma unroll
          for (int b = 0; b < T; ++b) dmma_8x8x4(acc[NG + a * T + b], p[a], u[b]);
    }
  }
  // the warps' sums in warp order
  for (int w = 0; w < NW; ++w) {
    if (warp == w)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double& r = red[t * 64 + 2 * lane + e];
          r = w == 0 ? acc[t][e] : r + acc[t][e];
        }
    __syncthreads();
  }
  for (int p = threadIdx.x; p < NT * 64; p += kGramThreads) out[p] = red[p];
  if (CROSS) store_stats(q, out + NT * 64);
  __syncthreads();
}

// The same for more than four column tiles (T at run time).
template <bool CROSS, bool SCALE>
__device__ __forceinline__ void gram_wide(const float* __restrict__ P, const float* __restrict__ U, uint64_t r0,
                                          uint64_t r1, int R, double* __restrict__ out, const GramScale& sc) {
  const int T = gram_tiles(R), NG = T * (T + 1) / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kr = lane & 3, kc = lane >> 2;
  double q[3] = {0.0, 0.0, 0.0};
  for (int a = warp; a < T; a += 8)
    for (int cb = 0; cb < T; cb += 8) {
      double g[8][2], c[CROSS ? 8 : 1][2];
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        g[b][0] = g[b][1] = 0.0;
        if (CROSS) c[b][0] = c[b][1] = 0.0;
      }
      double inv[SCALE ? 9 : 1];
      if constexpr (SCALE)
#pragma unroll
        for (int b = 0; b < 9; ++b) {
          const int col = (b < 8 ? cb + b : a) * 8 + kc;
          inv[b] = col < R ? 1.0 / sc.lambda[col] : 0.0;
        }
      float fb[8], fa = 0.f, pa = 0.f;
      auto fetch = [&](uint64_t k0) {
        const uint64_t row = k0 + kr;
        const bool in = row < r1;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const int col = (cb + b) * 8 + kc;
          fb[b] = in && col < R ? U[row * R + col] : 0.f;
        }
        const int col = a * 8 + kc;
        fa = in && col < R ? U[row * R + col] : 0.f;
        if (CROSS) pa = in && col < R ? P[row * R + col] : 0.f;
      };
      if (r0 < r1) fetch(r0);
      for (uint64_t k0 = r0; k0 < r1; k0 += 4) {
        double ub[8];
        if constexpr (SCALE) {
#pragma unroll
          for (int b = 0; b < 8; ++b) fb[b] = (float)((double)fb[b] * inv[b]);
          fa = (float)((double)fa * inv[8]);
          const uint64_t row = k0 + kr;
          const int col = a * 8 + kc;
          if (cb == 0 && row < r1 && col < R) {
            sc.Y[row * R + col] = fa;
            if (sc.shadow) sc.shadow[row * R + col] = __float2bfloat16(fa);
          }
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) ub[b] = (double)fb[b];
        const double ua = (double)fa, pv = (double)pa;
        if (k0 + 4 < r1) fetch(k0 + 4);
        if (CROSS && cb == 0) change_stats(pv, ua, q);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          if (cb + b >= a) dmma_8x8x4(g[b], ua, ub[b]);
          if (CROSS) dmma_8x8x4(c[b], pv, ub[b]);
        }
      }
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        if (cb + b >= T) continue;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (cb + b >= a) out[gram_tile_of(T, a, cb + b) * 64 + 2 * lane + e] = g[b][e];
          if (CROSS) out[(NG + a * T + cb + b) * 64 + 2 * lane + e] = c[b][e];
        }
      }
    }
  if (CROSS) store_stats(q, out + gram_out_tiles(T, true) * 64);
  __syncthreads();
}

// TT: 1 to 4 column tiles, or 0 for more.
template <int TT, bool CROSS, bool SCALE = false>
__device__ __forceinline__ void gram_block(const float* __restrict__ P, const float* __restrict__ U, uint64_t I, int R,
                                           uint64_t rows_per_block, double* __restrict__ partials, uint32_t block,
                                           const GramScale& sc = GramScale{}) {
  const uint64_t r0 = (uint64_t)block * rows_per_block;
  const uint64_t r1 = min(r0 + rows_per_block, I);
  double* out = partials + (size_t)block * gram_partial_len(R, CROSS);
  if constexpr (TT == 0)
    gram_wide<CROSS, SCALE>(P, U, r0, r1, R, out, sc);
  else
    gram_narrow<TT, CROSS, SCALE>(P, U, r0, r1, R, out, sc);
}

template <int TT>
struct GramLaunch {
  static constexpr int kThreads = TT ? kGramThreads : kGramThreadsWide;
  static constexpr int kMinBlocks = TT == 0 || TT == 4 ? 2 : 3;
};

template <int TT, bool CROSS>
__global__ void __launch_bounds__(GramLaunch<TT>::kThreads, GramLaunch<TT>::kMinBlocks)
    gram_kernel(const float* __restrict__ P, const float* __restrict__ U, uint64_t I, int R, uint64_t rows_per_block,
                double* __restrict__ partials) {
  gram_block<TT, CROSS>(P, U, I, R, rows_per_block, partials, blockIdx.x);
}

template <int TT>
__global__ void __launch_bounds__(GramLaunch<TT>::kThreads, GramLaunch<TT>::kMinBlocks)
    scale_gram_kernel(const float* __restrict__ U, uint64_t I, int R, uint64_t rows_per_block,
                      double* __restrict__ partials, GramScale sc) {
  gram_block<TT, false, true>(nullptr, U, I, R, rows_per_block, partials, blockIdx.x, sc);
}

// sum over blocks b of partials[b][p] for 32 consecutive p (one per lane), in a
// fixed order: warp w sums blocks w, w + nw, ... and the warp sums are added in
// warp order.  Every thread of warp 0 gets its p's sum.
constexpr int kReduceThreads = 512;
__host__ __device__ inline unsigned reduce_grid(int n) { return (unsigned)((n + 31) / 32); }

__device__ __forceinline__ double reduce_column(const double* __restrict__ partials, int nblocks, int n, int p) {
  __shared__ double s[kReduceThreads / 32][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double acc = 0.0;
  if (p < n)
#pragma unroll 4
    for (int b = w; b < nblocks; b += kReduceThreads / 32) acc += partials[(size_t)b * n + p];
  s[w][lane] = acc;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = s[0][lane];
    for (int k = 1; k < kReduceThreads / 32; ++k) t += s[k][lane];
  }
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(kReduceThreads)
    reduce_partials_kernel(const double* __restrict__ partials, int nblocks, int n, double* __restrict__ out) {
  const int p = blockIdx.x * 32 + (threadIdx.x & 31);
  const double t = reduce_column(partials, nblocks, n, p);
  if (threadIdx.x < 32 && p < n) out[p] = t;
}

// Reduction block `block` of a Gram pass: its outputs back in row-major order
// (G mirrored from the tiles on and above the diagonal).
template <bool CROSS>
__device__ __forceinline__ void gram_reduce_body(const double* __restrict__ partials, int nblocks, int R,
                                                 double* __restrict__ G, double* __restrict__ C,
                                                 double* __restrict__ stats3, uint32_t block) {
  const int n = gram_partial_len(R, CROSS), T = gram_tiles(R), NG = T * (T + 1) / 2, NT = gram_out_tiles(T, CROSS);
  const int p = block * 32 + (threadIdx.x & 31);
  const double t = reduce_column(partials, nblocks, n, p);
  if (threadIdx.x >= 32 || p >= n) return;
  if (p >= NT * 64) {
    if (stats3) stats3[p - NT * 64] = t;
    return;
  }
  int tile = p / 64;
  const int l = (p % 64) / 2, i = l >> 2, j = 2 * (l & 3) + (p & 1);
  if (tile < NG) {
    int a = 0;
    while (tile >= T - a) tile -= T - a++;
    const int row = a * 8 + i, col = (a + tile) * 8 + j;
    if (row >= R || col >= R) return;
    G[row * R + col] = t;
    if (tile) G[col * R + row] = t;
  } else {
    const int row = (tile - NG) / T * 8 + i, col = (tile - NG) % T * 8 + j;
    if (row < R && col < R) C[row * R + col] = t;
  }
}

template <bool CROSS>
__global__ void __launch_bounds__(kReduceThreads)
    gram_reduce_kernel(const double* __restrict__ partials, int nblocks, int R, double* __restrict__ G,
                       double* __restrict__ C, double* __restrict__ stats3) {
  gram_reduce_body<CROSS>(partials, nblocks, R, G, C, stats3, blockIdx.x);
}

// Grouped gram_cross_stats: partial blocks over all items (block_off
// prefix sums of the items' nb), then reduction blocks (red_off).
template <int TT>
__global__ void __launch_bounds__(GramLaunch<TT>::kThreads, GramLaunch<TT>::kMinBlocks)
    gram_group_partial_kernel(Strided<GramItem> items, const uint32_t* __restrict__ block_off, int R) {
  const int K = *items.count;
  const uint32_t total = K > 0 ? block_off[K] : 0;
  for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
    int lo = 0, hi = K;  // the last s with block_off[s] <= v
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (block_off[mid] <= v)
        lo = mid;
      else
        hi = mid;
    }
    const GramItem& it = items[lo];
    if (it.active && !*it.active) continue;
    gram_block<TT, true>(it.P, it.U, it.I, R, it.rpb, it.part, v - block_off[lo]);
  }
}

__global__ void __launch_bounds__(kReduceThreads)
    gram_group_reduce_kernel(Strided<GramItem> items, const uint32_t* __restrict__ red_off, int R) {
  const int K = *items.count;
  const uint32_t total = K > 0 ? red_off[K] : 0;
  for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
    int lo = 0, hi = K;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (red_off[mid] <= v)
        lo = mid;
      else
        hi = mid;
    }
    const GramItem& it = items[lo];
    if (it.active && !*it.active) continue;
    gram_reduce_body<true>(it.part, (int)it.nb, R, it.G, it.C, it.stats3, v - red_off[lo]);
  }
}

// At least 64 rows per block, at most kGramBlocksPerSm blocks per SM.
void gram_split(uint64_t I, uint32_t* nb_out, uint64_t* rpb_out) {
  uint64_t nb = std::min<uint64_t>((I + 63) / 64, (uint64_t)sms() * kGramBlocksPerSm);
  if (nb < 1) nb = 1;
  const uint64_t rpb = (I + nb - 1) / nb;
  nb = I ? (I + rpb - 1) / rpb : 1;
  *nb_out = (uint32_t)nb;
  *rpb_out = rpb;
}

uint64_t gram_partial_doubles(uint64_t I, int R, bool cross) {
  uint32_t nb = 1;
  uint64_t rpb = 1;
  gram_split(I, &nb, &rpb);
  return (uint64_t)nb * gram_partial_len(R, cross);
}

uint32_t gram_reduce_blocks(int R) { return reduce_grid(gram_partial_len(R, true)); }

// Launch `kernel<TT, ...>` for rank R.
#define GRAM_DISPATCH(R, LAUNCH) \
  switch (gram_tiles(R)) {       \
    case 1: LAUNCH(1); break;    \
    case 2: LAUNCH(2); break;    \
    case 3: LAUNCH(3); break;    \
    case 4: LAUNCH(4); break;    \
    default: LAUNCH(0); break;   \
  }

alto_status gram_group_launch(Strided<GramItem> items, const uint32_t* block_off, const uint32_t* red_off,
                              int max_items, int R, cudaStream_t st) {
  const unsigned grid = (unsigned)sms() * 3;
#define GG(TT) gram_group_partial_kernel<TT><<<grid, GramLaunch<TT>::kThreads, 0, st>>>(items, block_off, R)
  GRAM_DISPATCH(R, GG)
#undef GG
  ALTO_LAUNCHED();
  const unsigned rgrid = (unsigned)std::max(1, std::min(max_items * (int)gram_reduce_blocks(R), (int)sms() * 4));
  gram_group_reduce_kernel<<<rgrid, kReduceThreads, 0, st>>>(items, red_off, R);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

alto_status gram_cross_stats(const float* P, const float* U, uint64_t I, int R, double* G, double* C,
                             double* stats3, DevBuf& scratch, cudaStream_t st) {
  uint32_t nb = 1;
  uint64_t rpb = 1;
  gram_split(I, &nb, &rpb);
  ALTO_TRY(scratch.ensure(gram_partial_doubles(I, R, true) * sizeof(double)));
  double* part = scratch.as<double>();
  if (I == 0) {
    ALTO_TRY_CUDA(cudaMemsetAsync(part, 0, gram_partial_len(R, true) * sizeof(double), st));
  } else {
#define GC(TT) gram_kernel<TT, true><<<nb, GramLaunch<TT>::kThreads, 0, st>>>(P, U, I, R, rpb, part)
    GRAM_DISPATCH(R, GC)
#undef GC
    ALTO_LAUNCHED();
  }
  gram_reduce_kernel<true><<<gram_reduce_blocks(R), kReduceThreads, 0, st>>>(part, (int)nb, R, G, C, stats3);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// G = A^T A with nb partial results of rpb rows in `part`.
static alto_status gram_into(const float* A, uint64_t I, int R, uint32_t nb, uint64_t rpb, double* part, double* out,
                             cudaStream_t st) {
#define GP(TT) gram_kernel<TT, false><<<nb, GramLaunch<TT>::kThreads, 0, st>>>(nullptr, A, I, R, rpb, part)
  GRAM_DISPATCH(R, GP)
#undef GP
  ALTO_LAUNCHED();
  gram_reduce_kernel<false><<<reduce_grid(gram_partial_len(R, false)), kReduceThreads, 0, st>>>(part, (int)nb, R, out,
                                                                                              nullptr, nullptr);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

alto_status scale_gram(const float* X, uint64_t I, int R, const double* lambda, float* Y, __nv_bfloat16* shadow,
                       double* out, DevBuf& scratch, cudaStream_t st) {
  if (I == 0) {
    ALTO_TRY_CUDA(cudaMemsetAsync(out, 0, (size_t)R * R * sizeof(double), st));
    return ALTO_OK;
  }
  uint32_t nb = 1;
  uint64_t rpb = 1;
  gram_split(I, &nb, &rpb);
  ALTO_TRY(scratch.ensure(gram_partial_doubles(I, R, false) * sizeof(double)));
  double* part = scratch.as<double>();
  const GramScale sc{lambda, Y, shadow};
#define SG_LAUNCH(TT) scale_gram_kernel<TT><<<nb, GramLaunch<TT>::kThreads, 0, st>>>(X, I, R, rpb, part, sc)
  GRAM_DISPATCH(R, SG_LAUNCH)
#undef SG_LAUNCH
  ALTO_LAUNCHED();
  gram_reduce_kernel<false><<<reduce_grid(gram_partial_len(R, false)), kReduceThreads, 0, st>>>(part, (int)nb, R, out,
                                                                                              nullptr, nullptr);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

alto_status gram(const float* A, uint64_t I, int R, double* out, DevBuf& scratch, cudaStream_t st) {
  if (I == 0) {
    ALTO_TRY_CUDA(cudaMemsetAsync(out, 0, (size_t)R * R * sizeof(double), st));
    return ALTO_OK;
  }
  uint32_t nb = 1;
  uint64_t rpb = 1;
  gram_split(I, &nb, &rpb);
  ALTO_TRY(scratch.ensure(gram_partial_doubles(I, R, false) * sizeof(double)));
  return gram_into(A, I, R, nb, rpb, scratch.as<double>(), out, st);
}

// ------------------------------------------------------- R x R solve setup

// One CTA (ranks above 64): V = prod_{m in mask} G_m (elementwise), then per `kind`:
//   SOLVE_RIDGE: V += ridge * I;  ADMM: rho = tr(V)/R, V += rho * I.
// Cholesky of V (upper triangle read, as dpotrf 'L' on the column-major
// view); on success W = V^{-1}.  On failure: kind SOLVE_RIDGE_DIAG_FALLBACK
// writes the reference's dgelsy fallback for CP-ALS, W = diag(1/V_rr) of V
// without the ridge (include/cpd.hpp:436-476: its restored V has zero
// lower triangles mirrored over the upper one); kind kSolveRidgeKeep writes
// W = I (the right-hand side is left as it is); otherwise W = 0.
// status[0] = LAPACK-style info (0 = success), rho_out[0] = rho.
__global__ void solve_setup_kernel(const double* __restrict__ grams, int nmodes, unsigned mask,
                                   int R, int kind, double ridge, double* __restrict__ W,
                                   int* __restrict__ status, double* __restrict__ rho_out) {
  extern __shared__ double A[];  // R x R
  const int RR = R * R;
  for (int p = threadIdx.x; p < RR; p += blockDim.x) {
    double v = 1.0;
    for (int m = 0; m < nmodes; ++m)
      if (mask & (1u << m)) v *= grams[(size_t)m * RR + p];
    A[p] = v;
  }
  __syncthreads();
  __shared__ double s_rho;
  __shared__ int s_info;
  if (threadIdx.x == 0) {
    double add = ridge;
    if (kind == kSolveAdmm) {
      double tr = 0.0;
      for (int r = 0; r < R; ++r) tr += A[r * R + r];
      add = tr / (double)R;
    }
    s_rho = add;
    s_info = 0;
  }
  __syncthreads();
  // keep the unridged diagonal for the fallback in W's diagonal slots
  if (kind == kSolveRidgeDiagFallback)
    for (int r = threadIdx.x; r < R; r += blockDim.x) W[r * R + r] = A[r * R + r];
  for (int r = threadIdx.x; r < R; r += blockDim.x) A[r * R + r] += s_rho;
  __syncthreads();
  // right-looking Cholesky, lower factor in A's lower triangle (reads upper)
  for (int j = 0; j < R; ++j) {
    if (threadIdx.x == 0) {
      double d = A[j * R + j];
      for (int k = 0; k < j; ++k) d -= A[j * R + k] * A[j * R + k];
      if (!(d > 0.0)) {
        if (!s_info) s_info = j + 1;
        d = 1.0;
      }
      A[j * R + j] = sqrt(d);
    }
    __syncthreads();
    const double djj = A[j * R + j];
    for (int i = j + 1 + threadIdx.x; i < R; i += blockDim.x) {
      double s = A[j * R + i];
      for (int k = 0; k < j; ++k) s -= A[i * R + k] * A[j * R + k];
      A[i * R + j] = s / djj;
    }
    __syncthreads();
  }
  const int info = s_info;
  if (info) {
    for (int p = threadIdx.x; p < RR; p += blockDim.x) {
      const int a = p / R, b = p % R;
      if (kind == kSolveRidgeDiagFallback) {
        if (a != b) W[p] = 0.0;
      } else {
        W[p] = (kind == kSolveRidgeKeep && a == b) ? 1.0 : 0.0;
      }
    }
    __syncthreads();
    if (kind == kSolveRidgeDiagFallback)
      for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const double d = W[r * R + r];
        W[r * R + r] = d != 0.0 ? 1.0 / d : 0.0;
      }
  } else {
    // L^{-1} by forward substitution, one column per thread:
    // x_i = (delta_ic - sum_{k=c}^{i-1} L[i][k] x_k) / L[i][i], kept in row c of W.
    for (int c = threadIdx.x; c < R; c += blockDim.x) {
      double* x = W + (size_t)c * R;
      for (int i = 0; i < c; ++i) x[i] = 0.0;
      for (int i = c; i < R; ++i) {
        double s = (i == c) ? 1.0 : 0.0;
        for (int k = c; k < i; ++k) s -= A[i * R + k] * x[k];
        x[i] = s / A[i * R + i];
      }
    }
    __syncthreads();
    // W currently holds rows c = columns of L^{-1}: Linv[i][c] = W[c*R + i].
    // Copy L^{-1} into A (lower) then W[a][b] = sum_{k >= max(a,b)} Linv[k][a] Linv[k][b].
    for (int p = threadIdx.x; p < RR; p += blockDim.x) {
      const int c = p / R, i = p % R;
      if (i >= c) A[i * R + c] = W[(size_t)c * R + i];
    }
    __syncthreads();
    for (int p = threadIdx.x; p < RR; p += blockDim.x) {
      const int a = p / R, b = p % R;
      const int k0 = a > b ? a : b;
      double s = 0.0;
      for (int k = k0; k < R; ++k) s += A[k * R + a] * A[k * R + b];
      W[p] = s;
    }
  }
  if (threadIdx.x == 0) {
    status[0] = info;
    if (rho_out) rho_out[0] = s_rho;
  }
}

// The same set-up for R <= RMAX = 8, 16, 32 or 64, bound by the chain of R
// dependent pivots.  One warp factors a 32 x 32 block (RMAX x RMAX below 32)
// with lane i holding row i of the matrix and column i of L^-1 in registers: a
// column of L goes through shared memory once and updates both, and the next
// pivot's reciprocal square root is started before the rest of the update, so a
// step costs one rsqrt and one shared-memory round trip, with no block barrier.
// At RMAX 64 the two 32 x 32 diagonal blocks are factored so, and the rest of
// L^-1 and W = L^-T L^-1 are float64 tensor-core products of the block.  One
// thread per element with three to five barriers per column took 10.4 us at
// rank 16, 40 us at rank 32 and (one column at a time) 192 us at rank 64; now 6, 10 and
// 50 us.
// Matrices smaller than RMAX are extended by the identity.

// d += A B of one 8 x 8 tile over K (a multiple of 4): fa(i, k), fb(k, j) the
// operands, i and j in [0, 8); lane l gets (l / 4, 2 (l % 4)) and its right
// neighbour.
template <typename FA, typename FB>
__device__ __forceinline__ void dmma_tile(int K, int lane, FA fa, FB fb, double (&d)[2]) {
  for (int k = 0; k < K; k += 4) dmma_8x8x4(d, fa(lane >> 2, k + (lane & 3)), fb(k + (lane & 3), lane >> 2));
}

// One warp: the Cholesky factor L of the N x N block at A (leading dimension
// LD, shift added to the first `live` diagonal entries) and X = L^-1 (zero
// above the diagonal), N <= 32.  Returns the 1-based index of the first pivot
// that is not positive (0: none); col: 2 x 32 doubles of shared memory.
template <int N>
__device__ __forceinline__ int warp_chol_inverse(const double* A, int LD, double shift, int live, double* X, int LDX,
                                                 double* col, int lane) {
  double a[N], x[N];
  const int row = lane < N ? lane : N - 1;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    a[k] = A[row * LD + k] + (k == row && k < live ? shift : 0.0);
    x[k] = k == row ? 1.0 : 0.0;
  }
  int info = 0;
  double d = __shfl_sync(0xffffffffu, a[0], 0);
  if (!(d > 0.0)) {
    info = 1;
    d = 1.0;
  }
  double rs = rsqrt(d);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const double l = a[j] * rs;  // L[lane][j]
    double* c = col + (j & 1) * 32;
    c[lane] = l;
    __syncwarp();
    x[j] *= rs;
    double rs_next = 0.0;
    if (j + 1 < N) {
      const double l1 = c[j + 1];
      a[j + 1] = __fma_rn(-l, l1, a[j + 1]);
      x[j + 1] = __fma_rn(-l1, x[j], x[j + 1]);
      d = __shfl_sync(0xffffffffu, a[j + 1], j + 1);
      if (!(d > 0.0)) {
        if (!info) info = j + 2;
        d = 1.0;
      }
      rs_next = rsqrt(d);
    }
#pragma unroll
    for (int k = j + 2; k < N; ++k) {
      const double lk = c[k];
      a[k] = __fma_rn(-l, lk, a[k]);
      x[k] = __fma_rn(-lk, x[j], x[k]);
    }
    rs = rs_next;
  }
  if (lane < N)
#pragma unroll
    for (int k = 0; k < N; ++k) X[k * LDX + lane] = k >= lane ? x[k] : 0.0;
  return info;
}

template <int RMAX>
struct SetupCfg {
  static constexpr int LD = RMAX + (RMAX >= 32 ? 4 : 0);  // (tensor-core operand reads in fewer conflicts)
  static constexpr int kThreads = RMAX <= 16 ? 128 : 256;
  static constexpr size_t smem_bytes() { return 2 * (size_t)RMAX * LD * sizeof(double); }
};

template <int RMAX>
__device__ __forceinline__ void solve_setup_block_body(const double* __restrict__ grams, int nmodes, unsigned mask,
                                                       int R, int kind, double ridge, double* __restrict__ W,
                                                       int* __restrict__ status, double* __restrict__ rho_out) {
  constexpr int LD = SetupCfg<RMAX>::LD;
  constexpr int N = RMAX < 32 ? RMAX : 32;
  extern __shared__ __align__(16) double setup_smem[];
  double* A = setup_smem;
  double* X = A + RMAX * LD;
  __shared__ double s_col[64];
  __shared__ double s_rho;
  __shared__ int s_info[2];
  const int RR = R * R;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  for (int p = tid; p < RMAX * RMAX; p += blockDim.x) {
    const int a = p / RMAX, b = p % RMAX;
    double v = a == b ? 1.0 : 0.0;
    if (a < R && b < R) {
      v = 1.0;
      for (int m = 0; m < nmodes; ++m)
        if (mask & (1u << m)) v *= grams[(size_t)m * RR + a * R + b];
      if (kind == kSolveRidgeDiagFallback && a == b) W[a * R + a] = v;  // the unridged diagonal, for the fallback
    }
    A[a * LD + b] = v;
  }
  __syncthreads();
  if (warp == 0) {
    double add = ridge;
    if (kind == kSolveAdmm) {  // rho = tr(V) / R
      double tr = 0.0;
      for (int r = lane; r < R; r += 32) tr += A[r * LD + r];
      for (int o = 16; o; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
      add = tr / (double)R;
    }
    const int info = warp_chol_inverse<N>(A, LD, add, min(R, N), X, LD, s_col, lane);
    if (lane == 0) {
      s_rho = add;
      s_info[0] = info;
      s_info[1] = 0;
    }
  }
  __syncthreads();
  if constexpr (RMAX == 64) {
    // L21 = A21 X11^T over A21 (each warp its tiles; A12, the mirror, is free
    // and holds the product until every tile is done), A22 -= L21 L21^T
    constexpr int H = 32;
    double* A21 = A + H * LD;
    double* A12 = A + H;
    double* A22 = A + H * LD + H;
    double* X21 = X + H * LD;
    double* X22 = X + H * LD + H;
    const int i0 = lane >> 2, j0 = 2 * (lane & 3);
    for (int q = warp; q < 16; q += nw) {
      const int ti = (q >> 2) * 8, tj = (q & 3) * 8;
      double d[2] = {0.0, 0.0};
      dmma_tile(H, lane, [&](int i, int k) { return A21[(ti + i) * LD + k]; },
                [&](int k, int j) { return X[(tj + j) * LD + k]; }, d);
      A12[(ti + i0) * LD + tj + j0] = d[0];
      A12[(ti + i0) * LD + tj + j0 + 1] = d[1];
    }
    __syncthreads();
    const double* L21 = A12;
    for (int q = warp; q < 16; q += nw) {
      const int ti = (q >> 2) * 8, tj = (q & 3) * 8;
      double d[2] = {0.0, 0.0};
      dmma_tile(H, lane, [&](int i, int k) { return L21[(ti + i) * LD + k]; },
                [&](int k, int j) { return L21[(tj + j) * LD + k]; }, d);
      A22[(ti + i0) * LD + tj + j0] -= d[0];
      A22[(ti + i0) * LD + tj + j0 + 1] -= d[1];
      // T = L21 X11 over A21
      double t[2] = {0.0, 0.0};
      dmma_tile(H, lane, [&](int i, int k) { return L21[(ti + i) * LD + k]; },
                [&](int k, int j) { return X[k * LD + tj + j]; }, t);
      A21[(ti + i0) * LD + tj + j0] = t[0];
      A21[(ti + i0) * LD + tj + j0 + 1] = t[1];
      X[(ti + i0) * LD + H + tj + j0] = 0.0;  // above the diagonal
      X[(ti + i0) * LD + H + tj + j0 + 1] = 0.0;
    }
    __syncthreads();
    if (warp == 0) {
      const int info = warp_chol_inverse<H>(A22, LD, s_rho, max(R - H, 0), X22, LD, s_col, lane);
      if (lane == 0 && info) s_info[1] = H + info;
    }
    __syncthreads();
    for (int q = warp; q < 16; q += nw) {  // X21 = -X22 T
      const int ti = (q >> 2) * 8, tj = (q & 3) * 8;
      double d[2] = {0.0, 0.0};
      dmma_tile(H, lane, [&](int i, int k) { return X22[(ti + i) * LD + k]; },
                [&](int k, int j) { return A21[k * LD + tj + j]; }, d);
      X21[(ti + i0) * LD + tj + j0] = -d[0];
      X21[(ti + i0) * LD + tj + j0 + 1] = -d[1];
    }
    __syncthreads();
  }
  const int info = s_info[0] ? s_info[0] : s_info[1];
  if (info) {
    for (int p = tid; p < RR; p += blockDim.x) {
      const int a = p / R, b = p % R;
      if (kind == kSolveRidgeDiagFallback) {
        const double dv = a == b ? W[p] : 0.0;
        W[p] = dv != 0.0 ? 1.0 / dv : 0.0;
      } else {
        W[p] = (kind == kSolveRidgeKeep && a == b) ? 1.0 : 0.0;
      }
    }
  } else {
    // W = X^T X (X is zero above its diagonal): 8 x 8 tiles on and above the
    // diagonal, mirrored
    constexpr int T = RMAX / 8;
    for (int q = warp; q < T * T; q += nw) {
      const int ti = (q / T) * 8, tj = (q % T) * 8;
      if (tj < ti) continue;
      double d[2] = {0.0, 0.0};
      dmma_tile(RMAX - tj, lane, [&](int i, int k) { return X[(tj + k) * LD + ti + i]; },
                [&](int k, int j) { return X[(tj + k) * LD + tj + j]; }, d);
      const int a = ti + (lane >> 2);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int b = tj + 2 * (lane & 3) + e;
        if (a < R && b < R) {
          W[a * R + b] = d[e];
          if (ti != tj) W[b * R + a] = d[e];
        }
      }
    }
  }
  if (tid == 0) {
    status[0] = info;
    if (rho_out) rho_out[0] = s_rho;
  }
  __syncthreads();
}

template <int RMAX>
__global__ void __launch_bounds__(SetupCfg<RMAX>::kThreads)
    solve_setup_block_kernel(const double* __restrict__ grams, int nmodes, unsigned mask, int R, int kind,
                             double ridge, double* __restrict__ W, int* __restrict__ status,
                             double* __restrict__ rho_out) {
  solve_setup_block_body<RMAX>(grams, nmodes, mask, R, kind, ridge, W, status, rho_out);
}

// One CTA per item in turn (R <= 32).
template <int RMAX>
__global__ void __launch_bounds__(SetupCfg<RMAX>::kThreads) setup_group_kernel(Strided<SetupItem> items, int R) {
  const int K = *items.count;
  for (int s = blockIdx.x; s < K; s += gridDim.x) {
    const SetupItem& it = items[s];
    if (it.active && !*it.active) continue;
    solve_setup_block_body<RMAX>(it.grams, it.nmodes, it.mask, R, it.kind, it.ridge, it.W, it.status, it.rho);
  }
}

alto_status setup_group_launch(Strided<SetupItem> items, int max_items, int R, cudaStream_t st) {
  const unsigned grid = (unsigned)std::max(1, std::min(max_items, 1024));
  if (R <= 8)
    setup_group_kernel<8><<<grid, SetupCfg<8>::kThreads, SetupCfg<8>::smem_bytes(), st>>>(items, R);
  else if (R <= 16)
    setup_group_kernel<16><<<grid, SetupCfg<16>::kThreads, SetupCfg<16>::smem_bytes(), st>>>(items, R);
  else if (R <= 32)
    setup_group_kernel<32><<<grid, SetupCfg<32>::kThreads, SetupCfg<32>::smem_bytes(), st>>>(items, R);
  else {
    set_error("grouped solve set-up takes rank <= 32 (got %d)", R);
    return ALTO_ERR_UNSUPPORTED;
  }
  ALTO_LAUNCHED();
  return ALTO_OK;
}

alto_status solve_setup(const double* grams, int nmodes, unsigned mask, int R, int kind,
                        double ridge, double* W, int* status, double* rho, cudaStream_t st) {
#define SETUP_CASE(RM)                                                                                        \
  if (R <= RM) {                                                                                              \
    solve_setup_block_kernel<RM><<<1, SetupCfg<RM>::kThreads, SetupCfg<RM>::smem_bytes(), st>>>(              \
        grams, nmodes, mask, R, kind, ridge, W, status, rho);                                                 \
    ALTO_LAUNCHED();                                                                                          \
    return ALTO_OK;                                                                                           \
  }
  SETUP_CASE(8)
  SETUP_CASE(16)
  SETUP_CASE(32)
  if (R <= 64) {  // (the shared-memory limit is raised once per device, outside any capture)
    static std::atomic<bool> raised64[64];
    int dev = 0;
    ALTO_TRY_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !raised64[dev].load()) {
      ALTO_TRY_CUDA(cudaFuncSetAttribute(solve_setup_block_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)SetupCfg<64>::smem_bytes()));
      if (dev >= 0 && dev < 64) raised64[dev] = true;
    }
  }
  SETUP_CASE(64)
#undef SETUP_CASE
  const size_t smem = (size_t)R * R * sizeof(double);
  static size_t raised = 0;
  if (smem > 48 * 1024 && smem > raised) {
    ALTO_TRY_CUDA(cudaFuncSetAttribute(solve_setup_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    raised = smem;
  }
  solve_setup_kernel<<<1, 256, smem, st>>>(grams, nmodes, mask, R, kind, ridge, W, status, rho);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// ------------------------------------------------------------ row apply
//
// X = B W (float32 in and out, float64 products) and the column scales of
// CP-ALS's normalisation, lambda[c] = sqrt(max(sum x^2, 1e-12)) (which 0) or
// max(1, max x) (which 1) over the float32 results.  Rows in registers as in
// alto_dmma.cuh (8 T columns; the columns past R are zero); each block leaves
// its columns' partial statistics and the last block to finish combines them in
// block order, so no launch of its own waits for them.  Bound by latency at
// CP-ALS's sizes: a shuffle per term and a one-block pass over every block's
// statistics took 50 + 17 us for up to 20,000 rows at rank 64 (now 14), 10 + 3 us
// for 1000 rows at rank 16.
constexpr int kApplyThreads = 256;

template <int T>
__device__ __forceinline__ void apply_rows(const float* __restrict__ B, uint64_t row, bool in, int quad, int R,
                                           float (&b)[T][2]) {
#pragma unroll
  for (int c = 0; c < T; ++c) {
    const int col = 8 * c + 2 * quad;
    if ((R & 1) == 0) {
      float2 v = make_float2(0.f, 0.f);
      if (in && col < R) v = *reinterpret_cast<const float2*>(B + row * R + col);
      b[c][0] = v.x;
      b[c][1] = v.y;
    } else {
      b[c][0] = in && col < R ? B[row * R + col] : 0.f;
      b[c][1] = in && col + 1 < R ? B[row * R + col + 1] : 0.f;
    }
  }
}

template <int T>
__global__ void __launch_bounds__(kApplyThreads)
    apply_kernel(const float* __restrict__ B, const double* __restrict__ W, uint64_t I, int R, float* __restrict__ X,
                 int which, double* __restrict__ partials, unsigned* __restrict__ ticket,
                 double* __restrict__ lambda) {
  constexpr int NW = kApplyThreads / 32;
  constexpr int NC = T < 4 ? T : 4;  // column tiles of a product at once
  extern __shared__ double sfrag[];
  __shared__ double sred[NW][8 * T];
  __shared__ bool last;
  load_fragments(sfrag, W, R, T);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quad = lane & 3;
  double acc[T][2];
#pragma unroll
  for (int c = 0; c < T; ++c) acc[c][0] = acc[c][1] = which ? -INFINITY : 0.0;
  for (uint64_t r0 = (uint64_t)blockIdx.x * 8 * NW + 8 * warp; r0 < I; r0 += (uint64_t)gridDim.x * 8 * NW) {
    const uint64_t row = r0 + (lane >> 2);
    const bool in = row < I;
    float b[T][2];
    apply_rows<T>(B, row, in, quad, R, b);
#pragma unroll
    for (int n0 = 0; n0 < T; n0 += NC) {
      double x[NC][2];
#pragma unroll
      for (int n = 0; n < NC; ++n) x[n][0] = x[n][1] = 0.0;
#pragma unroll
      for (int c = 0; c < T; ++c)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double a = (double)b[c][e];
#pragma unroll
          for (int n = 0; n < NC; ++n)
            if (n0 + n < T) dmma_8x8x4(x[n], a, sfrag[((c * 2 + e) * T + n0 + n) * 32 + lane]);
        }
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        if (n0 + n >= T) continue;
        const int col = 8 * (n0 + n) + 2 * quad;
        const float f[2] = {(float)x[n][0], (float)x[n][1]};
        if (!in) continue;
        if ((R & 1) == 0) {
          if (col < R) *reinterpret_cast<float2*>(X + row * R + col) = make_float2(f[0], f[1]);
        } else {
          if (col < R) X[row * R + col] = f[0];
          if (col + 1 < R) X[row * R + col + 1] = f[1];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double v = (double)f[e];
          acc[n0 + n][e] = which ? fmax(acc[n0 + n][e], v) : __fma_rn(v, v, acc[n0 + n][e]);
        }
      }
    }
  }
  // columns: the eight rows of a warp, the warps, the blocks, each in order
#pragma unroll
  for (int c = 0; c < T; ++c)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      double v = acc[c][e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, v, o);
        v = which ? fmax(v, y) : v + y;
      }
      if (lane < 4) sred[warp][8 * c + 2 * lane + e] = v;
    }
  __syncthreads();
  for (int r = threadIdx.x; r < 8 * T; r += kApplyThreads) {
    double v = sred[0][r];
    for (int w = 1; w < NW; ++w) v = which ? fmax(v, sred[w][r]) : v + sred[w][r];
    partials[(size_t)blockIdx.x * 8 * T + r] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  constexpr int kGroups = kApplyThreads / (8 * T) < NW ? kApplyThreads / (8 * T) : NW;  // threads per column
  const int r = threadIdx.x % (8 * T), g = threadIdx.x / (8 * T);
  if (g < kGroups) {
    double v = which ? -INFINITY : 0.0;
#pragma unroll 8
    for (unsigned b = g; b < gridDim.x; b += kGroups) {
      const double y = __ldcg(partials + (size_t)b * 8 * T + r);
      v = which ? fmax(v, y) : v + y;
    }
    sred[g][r] = v;
  }
  __syncthreads();
  if (threadIdx.x < R) {
    double v = sred[0][threadIdx.x];
    for (int k = 1; k < kGroups; ++k) v = which ? fmax(v, sred[k][threadIdx.x]) : v + sred[k][threadIdx.x];
    lambda[threadIdx.x] = which ? fmax(1.0, v) : sqrt(v > 1e-12 ? v : 1e-12);
  }
  if (threadIdx.x == 0) *ticket = 0;
}

// One block per SM at most: the last block reads every block's statistics.
static unsigned apply_blocks(uint64_t I) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((I + 63) / 64, (uint64_t)sms()));
}

template <int T>
static alto_status apply_launch(const float* B, const double* W, uint64_t I, int R, float* X, int which,
                                double* partials, unsigned* ticket, double* lambda, cudaStream_t st) {
  const size_t smem = (size_t)64 * T * T * sizeof(double);
  if (smem > 40 * 1024) {
    static std::atomic<bool> raised[64];  // per device
    int dev = 0;
    ALTO_TRY_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !raised[dev].load()) {
      ALTO_TRY_CUDA(cudaFuncSetAttribute(apply_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      if (dev >= 0 && dev < 64) raised[dev] = true;
    }
  }
  apply_kernel<T><<<apply_blocks(I), kApplyThreads, smem, st>>>(B, W, I, R, X, which, partials, ticket, lambda);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

size_t apply_scratch_bytes(uint64_t I, int R) { return 256 + (size_t)apply_blocks(I) * 8 * 16 * sizeof(double); }

alto_status apply_lambda(const float* B, const double* W, uint64_t I, int R, float* X, int which, void* scratch,
                         double* lambda, cudaStream_t st) {
  unsigned* ticket = static_cast<unsigned*>(scratch);
  double* part = reinterpret_cast<double*>(static_cast<char*>(scratch) + 256);
  const int T = gram_tiles(R);
#define APPLY_CASE(TT) \
  if (T <= TT) return apply_launch<TT>(B, W, I, R, X, which, part, ticket, lambda, st);
  APPLY_CASE(1)
  APPLY_CASE(2)
  APPLY_CASE(3)
  APPLY_CASE(4)
  APPLY_CASE(8)
  APPLY_CASE(16)
#undef APPLY_CASE
  set_error("rank %d is not supported", R);
  return ALTO_ERR_UNSUPPORTED;
}

// ----------------------------------------------------------- normalisation

// X[i][r] /= lambda[r]; optional bfloat16 shadow copy.
__global__ void scale_kernel(float* __restrict__ X, uint64_t n, int R,
                             const double* __restrict__ lambda, __nv_bfloat16* __restrict__ shadow) {
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const float v = (float)((double)X[q] / lambda[q % R]);
    X[q] = v;
    if (shadow) shadow[q] = __float2bfloat16(v);
  }
}

alto_status scale_columns(float* X, uint64_t I, int R, const double* lambda, __nv_bfloat16* shadow,
                          cudaStream_t st) {
  const uint64_t n = I * R;
  if (!n) return ALTO_OK;
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sms() * 8);
  scale_kernel<<<grid, 256, 0, st>>>(X, n, R, lambda, shadow);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

__global__ void to_bf16_kernel(const float* __restrict__ X, uint64_t n, __nv_bfloat16* __restrict__ Y) {
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n;
       q += (uint64_t)gridDim.x * blockDim.x)
    Y[q] = __float2bfloat16(X[q]);
}

alto_status to_bf16(const float* X, uint64_t n, __nv_bfloat16* Y, cudaStream_t st) {
  if (!n) return ALTO_OK;
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)sms() * 8);
  to_bf16_kernel<<<grid, 256, 0, st>>>(X, n, Y);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// ------------------------------------------------------------ reductions

// Per-block partial sums of up to 4 quantities over n elements:
//   q0 = sum a*b (dot), q1 = sum (a-b)^2, q2 = sum b^2.
template <typename TA, typename TB>
__global__ void __launch_bounds__(256)
    dot_partial_kernel(const TA* __restrict__ a, const TB* __restrict__ b, uint64_t n,
                       const double* __restrict__ colw, int R, double* __restrict__ partials) {
  double q0 = 0, q1 = 0, q2 = 0;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n;
       q += (uint64_t)gridDim.x * blockDim.x) {
    const double x = (double)a[q], y = (double)b[q];
    const double w = colw ? colw[q % R] : 1.0;
    q0 += x * y * w;
    q1 += (x - y) * (x - y);
    q2 += y * y;
  }
  __shared__ double s[3][8];
  for (int o = 16; o; o >>= 1) {
    q0 += __shfl_xor_sync(0xffffffffu, q0, o);
    q1 += __shfl_xor_sync(0xffffffffu, q1, o);
    q2 += __shfl_xor_sync(0xffffffffu, q2, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s[0][warp] = q0;
    s[1][warp] = q1;
    s[2][warp] = q2;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[threadIdx.x][w];
    partials[(size_t)blockIdx.x * 3 + threadIdx.x] = t;
  }
}

static constexpr int kDotBlocks = 296;

size_t dot_scratch_bytes() { return kDotBlocks * 3 * sizeof(double); }

alto_status dot_stats(const float* a, const float* b, uint64_t n, const double* colw, int R,
                      double* out3, DevBuf& scratch, cudaStream_t st) {
  ALTO_TRY(scratch.ensure(dot_scratch_bytes()));
  dot_partial_kernel<float, float><<<kDotBlocks, 256, 0, st>>>(a, b, n, colw, R, scratch.as<double>());
  ALTO_LAUNCHED();
  reduce_partials_kernel<<<reduce_grid(3), kReduceThreads, 0, st>>>(scratch.as<double>(), kDotBlocks, 3, out3);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// Sum of squares of n float values (||X||^2 of the tensor values).
__global__ void sumsq_partial_kernel(const float* __restrict__ v, uint64_t n, double* __restrict__ part) {
  double s = 0;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < n;
       q += (uint64_t)gridDim.x * blockDim.x)
    s += (double)v[q] * (double)v[q];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double w[8];
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += w[k];
    part[blockIdx.x] = t;
  }
}

alto_status sum_squares(const float* v, uint64_t n, double* out, DevBuf& scratch, cudaStream_t st) {
  ALTO_TRY(scratch.ensure(kDotBlocks * sizeof(double)));
  sumsq_partial_kernel<<<kDotBlocks, 256, 0, st>>>(v, n, scratch.as<double>());
  ALTO_LAUNCHED();
  reduce_partials_kernel<<<reduce_grid(1), kReduceThreads, 0, st>>>(scratch.as<double>(), kDotBlocks, 1, out);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// CP-ALS model norm from Grams and lambda (include/cpd.hpp:221-256):
// reference mode keeps the diagonal only; exact mode the whole product.
__global__ void model_norm_kernel(const double* __restrict__ grams, int nmodes, int R,
                                  const double* __restrict__ lambda, int exact,
                                  double* __restrict__ out) {
  __shared__ double part[32];
  double s = 0.0;
  const int RR = R * R;
  for (int p = threadIdx.x; p < RR; p += blockDim.x) {
    const int a = p / R, b = p % R;
    if (b > a) continue;
    if (!exact && a != b) continue;
    double t = lambda[a] * lambda[b];
    for (int m = 0; m < nmodes; ++m) t *= grams[(size_t)m * RR + p];
    s += (a == b) ? t : 2.0 * t;
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += part[k];
    out[0] = fabs(t);
  }
}

alto_status model_norm(const double* grams, int nmodes, int R, const double* lambda, int exact,
                       double* out, cudaStream_t st) {
  model_norm_kernel<<<1, R > 16 ? 1024 : 256, 0, st>>>(grams, nmodes, R, lambda, exact, out);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// Small elementwise R x R helpers.
__global__ void rr_kernel(double* __restrict__ dst, const double* __restrict__ a,
                          const double* __restrict__ b, int n, int op, double alpha) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    if (op == 0) dst[p] = a[p];              // copy
    else if (op == 1) dst[p] *= a[p];        // hadamard in place
    else if (op == 2) dst[p] *= alpha;       // scale
    else if (op == 3) dst[p] = 0.0;          // zero
  }
}

alto_status rr_op(double* dst, const double* a, int n, int op, double alpha, cudaStream_t st) {
  rr_kernel<<<(n + 255) / 256, 256, 0, st>>>(dst, a, nullptr, n, op, alpha);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// G += sum over rows of s s^T (the time-mode Gram update,
// src/streaming_cpd.cpp:1320-1327), s float64 rows.
__global__ void rank_update_kernel(double* __restrict__ G, const double* __restrict__ S,
                                   uint64_t rows, int R) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < R * R; p += gridDim.x * blockDim.x) {
    const int a = p / R, b = p % R;
    double s = G[p];
    for (uint64_t q = 0; q < rows; ++q) s += S[q * R + b] * S[q * R + a];
    G[p] = s;
  }
}

alto_status rank_update(double* G, const double* S, uint64_t rows, int R, cudaStream_t st) {
  rank_update_kernel<<<(R * R + 255) / 256, 256, 0, st>>>(G, S, rows, R);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

}  // namespace alto

extern "C" alto_status alto_gram(const float* U, uint64_t rows, int rank, double* G,
                                 alto_cuda_stream stream) {
  if (!G || (rows && !U)) {
    alto::set_error("U or G is NULL");
    return ALTO_ERR_INVALID;
  }
  if (rank < 1 || rank > 128) {
    alto::set_error("rank %d outside 1..128", rank);
    return ALTO_ERR_UNSUPPORTED;
  }
  static thread_local alto::DevBuf* partials = new alto::DevBuf();
  return alto::gram(U, rows, rank, G, *partials, (cudaStream_t)stream);
}

// ------------------------------------------------ Gram without allocation
//
// Some callers cannot allocate device memory: code running under a memory
// pool or arena that owns every byte of the device (a serving process that
// pre-reserves HBM), callers whose allocator is forbidden inside a CUDA
// graph capture or a real-time loop, and embedders that must not call
// cudaMalloc / cudaFree at all.  alto_gram_noalloc gives them the Gram
// kernel with its scratch -- the per-block partial sums -- in a fixed
// device array that this library owns for the life of the process, on
// every GPU that loads it.
namespace {

constexpr int kNoAllocBlocks = 64;    // partial sums, one R x R block each
constexpr int kNoAllocMaxRank = 64;   // 64 blocks x 64 x 64 doubles = 2 MiB (a partial result is 36 of its 64 tiles)
static __device__ __align__(256) double g_gram_noalloc_scratch[kNoAllocBlocks * kNoAllocMaxRank *
                                                               kNoAllocMaxRank];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};

// Device address of the scratch array on the current device, resolved once
// per device (the array's name in host code is only a stand-in).  The
// address is kept for the process's life: a cudaDeviceReset of the device
// would leave it stale, which the header rules out for callers.
alto_status noalloc_scratch(double** out) {
  int dev = 0;
  ALTO_TRY_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) {
    alto::set_error("device ordinal %d beyond %d", dev, kNoAllocMaxDevices);
    return ALTO_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    ALTO_TRY_CUDA(cudaGetSymbolAddress(&p, g_gram_noalloc_scratch));
    g_noalloc_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return ALTO_OK;
}

}  // namespace

extern "C" alto_status alto_gram_noalloc(const float* U, uint64_t rows, int rank, double* G,
                                         alto_cuda_stream stream) {
  if (!G || (rows && !U)) {
    alto::set_error("U or G is NULL");
    return ALTO_ERR_INVALID;
  }
  if (rank < 1 || rank > kNoAllocMaxRank) {
    alto::set_error("alto_gram_noalloc: rank %d outside 1..%d (its fixed scratch holds %d partial "
                    "Grams of at most %d x %d doubles)", rank, kNoAllocMaxRank, kNoAllocBlocks,
                    kNoAllocMaxRank, kNoAllocMaxRank);
    return ALTO_ERR_UNSUPPORTED;
  }
  double* part = nullptr;
  ALTO_TRY(noalloc_scratch(&part));
  cudaStream_t st = (cudaStream_t)stream;
  if (rows == 0) {
    ALTO_TRY_CUDA(cudaMemsetAsync(G, 0, (size_t)rank * rank * sizeof(double), st));
    return ALTO_OK;
  }
  uint64_t nb = std::min<uint64_t>((rows + 63) / 64, (uint64_t)kNoAllocBlocks);
  const uint64_t rpb = (rows + nb - 1) / nb;
  nb = (rows + rpb - 1) / rpb;
  // every block writes its whole partial result, so no clearing is needed
  return alto::gram_into(U, rows, rank, (uint32_t)nb, rpb, part, G, st);
}
