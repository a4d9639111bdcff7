// ALTO MTTKRP on the device.
//
// Reference: mttkrp_alto_par and its variants (jeewhanchoi/ALTO-stream
// include/alto.hpp:826-908 dispatch, :1349-1407 atomic, :1544-1634
// da_mem_pull, :1636-1706 stream, :1708-1801 op_sched).  For every nonzero
// x = (i_0..i_{N-1}, v) of the line:  out[i_n, :] += v * prod_{m != n} U_m[i_m, :].
//
// Device design.  The line is cut into tiles of tile_nnz nonzeros (the
// reference's partitions, sized for the GPU); a persistent grid, sized by
// occupancy, walks the tiles, and each warp takes an equal chunk of a tile.
// Inside a warp, G lanes own one nonzero (each lane 4 rank elements, one 16-byte
// load per factor row, or 8 in two loads: LaneWidth, WalkCfg), and the warp's chunk is split
// into 32/G contiguous sub-ranges, one per lane group.  A group walks its
// sub-range in line order, two nonzeros per iteration with all their keys,
// values and factor rows loaded before any product is formed, and keeps the
// running sum of the current output row in registers: each run of equal
// rows costs one update, with no cross-lane traffic.  Updates go
//   * to shared memory, when the tile's output interval (rows between its
//     smallest and largest target index, the reference's prtn_intervals)
//     fits the staging buffer -- the reference's da_mem, on chip -- and the
//     staged rows are flushed once per tile with vector atomics (STAGED;
//     the single-row output of the stream mode is its degenerate case); or
//   * to global memory with 16-byte vector atomics (red.global.add.v4.f32),
//     the reference's atomic variant (ATOMIC); or
//   * (SORTED) the walk runs over a per-mode copy of the line ordered by the
//     output row (ALTO order among equal rows), so every run of a row is
//     contiguous, reduces in registers, and is written once per warp chunk --
//     the reference's op_sched traversal, materialised.  The copies of 3- to
//     5-mode lines hold their rows decoded and have a walk of their own
//     (walk_kernel).
// ALTO_MTTKRP_AUTO uses the autotuned choice when alto_mttkrp_autotune has
// measured one, else a rule on the tile intervals and the mode's reuse.
#include <algorithm>

#include "alto_group.cuh"

namespace alto {

constexpr uint32_t kNoRow = 0xffffffffu;
constexpr int kMttkrpThreads = 256;
constexpr int kMttkrpWarps = kMttkrpThreads / 32;
constexpr int kStageBytes = 96 * 1024;

template <typename FT>
__device__ __forceinline__ float4 load4(const void* base, size_t off);

template <>
__device__ __forceinline__ float4 load4<float>(const void* base, size_t off) {
  return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + off));
}

template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const void* base, size_t off) {
  uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(base) + off));
  float4 r;
  r.x = __uint_as_float(u.x << 16);
  r.y = __uint_as_float(u.x & 0xffff0000u);
  r.z = __uint_as_float(u.y << 16);
  r.w = __uint_as_float(u.y & 0xffff0000u);
  return r;
}


// Decode one mode's field from the line key held as 32-bit words
// w0..w3 (w0 lowest): a funnel shift of the two words the field starts in.
// Fields are at most 32 bits wide (mode lengths below 2^32).
__device__ __forceinline__ uint32_t field32(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int pos,
                                            uint32_t mask) {
  const int s = pos & 31;
  uint32_t v;
  switch (pos >> 5) {
    case 0: v = __funnelshift_r(w0, w1, s); break;
    case 1: v = __funnelshift_r(w1, w2, s); break;
    case 2: v = __funnelshift_r(w2, w3, s); break;
    default: v = w3 >> s; break;
  }
  return v & mask;
}

// Row of mode m of a record held as words w (the field of the
// mode-contiguous key).
__device__ __forceinline__ uint32_t rec_row(const uint32_t (&w)[4], const LineDecode& dec, int m) {
  return field32(w[0], w[1], w[2], w[3], dec.pos[m], (uint32_t)dec.mask[m]);
}

// This lane's V floats of a factor row: V/4 float4 pieces at columns
// q*4G + 4*sub (q = 0..V/4-1), so that one load instruction of the G lanes of
// a group reads 4G contiguous floats (whole 32-byte sectors).
template <typename FT, int V, int G>
__device__ __forceinline__ void load_row(const void* base, size_t row_off, int sub, float (&x)[V]) {
#pragma unroll
  for (int q = 0; q < V / 4; ++q) {
    const float4 f = load4<FT>(base, row_off + q * 4 * G + sub * 4);
    x[q * 4 + 0] = f.x;
    x[q * 4 + 1] = f.y;
    x[q * 4 + 2] = f.z;
    x[q * 4 + 3] = f.w;
  }
}

// One update of output row `row` with this lane's V floats.
template <int R, int V, int G>
__device__ __forceinline__ void flush_row(bool staged, float* smem, uint32_t iv_start, float* out,
                                          uint32_t row, int sub, const float (&acc)[V]) {
  if (staged) {
    float* s = smem + (size_t)(row - iv_start) * R + sub * 4;
#pragma unroll
    for (int q = 0; q < V / 4; ++q)
#pragma unroll
      for (int k = 0; k < 4; ++k) atomicAdd(s + q * 4 * G + k, acc[q * 4 + k]);
  } else {
    float* o = out + (size_t)row * R + sub * 4;
#pragma unroll
    for (int q = 0; q < V / 4; ++q)
      atomicAdd(reinterpret_cast<float4*>(o + q * 4 * G),
                make_float4(acc[q * 4], acc[q * 4 + 1], acc[q * 4 + 2], acc[q * 4 + 3]));
  }
}

// Floats per lane for rank R: 4, so the G = R/4 lanes of a group read one
// factor row with one 16-byte load each -- whole 128-byte lines at R = 32,
// which keeps the L1 data pipe at one wavefront per row.
template <int R>
struct LaneWidth {
  static constexpr int V = 4;
  static constexpr int G = R / V;     // lanes per nonzero
  static constexpr int NPW = 32 / G;  // groups (nonzeros in flight) per warp
};

// Keys and values of U consecutive line records, from global memory or
// from the line tile staged in shared memory (SMEM): one 16-byte load per
// record (two when the key needs more than 96 bits, HW == 2).
template <int HW, int U, bool SMEM>
__device__ __forceinline__ void load_keys(const void* line, uint32_t i0, uint32_t ge,
                                          uint32_t (&w)[U][4], float (&v)[U], bool (&valid)[U]) {
  const uint4* q = static_cast<const uint4*>(line);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t i = i0 + u;
    valid[u] = i < ge;
    uint4 a = make_uint4(0, 0, 0, 0), b = make_uint4(0, 0, 0, 0);
    if (valid[u]) {
      if (HW == 2) {
        a = SMEM ? q[2 * i] : __ldg(q + 2 * i);
        b = SMEM ? q[2 * i + 1] : __ldg(q + 2 * i + 1);
      } else {
        a = SMEM ? q[i] : __ldg(q + i);
      }
    }
    w[u][0] = a.x;
    w[u][1] = a.y;
    if (HW == 2) {
      w[u][2] = a.z;
      w[u][3] = a.w;
      v[u] = __uint_as_float(b.x);
    } else {
      w[u][2] = a.z;
      w[u][3] = 0;
      v[u] = __uint_as_float(a.w);
    }
  }
}

// Walk line range [ws, we) with one warp: the range is split into NPW
// contiguous sub-ranges, one per lane group; a group walks its sub-range in
// order, U nonzeros per iteration (two for 3 modes, one for more, to stay in
// registers), with the next iteration's keys loaded while this iteration's
// factor rows are in flight; it keeps the running sum of the current output
// row in registers and updates the output once per run of equal rows.  NM is
// the mode count (3, 4, 5 specialised as in the reference's
// ALTO_MODES_SPECIALIZED, 8 for the rest).
// Deterministic mode (DET): the line is ordered by the target row, so a run
// that is neither the first nor the last of its sub-range holds every
// nonzero of its row and is added to the output without atomics; the first
// and last runs go to the sub-range's two slots (sub-range `sr`) and are
// summed in slot order by det_fix_*.
template <int R, int V, int G>
__device__ __forceinline__ void det_slot(const MttkrpArgs& a, uint32_t slot, uint32_t row, int sub,
                                         const float (&acc)[V], bool zero) {
  if (sub == 0) a.det_rows[slot] = row;
#pragma unroll
  for (int q = 0; q < V / 4; ++q)
    *reinterpret_cast<float4*>(a.det_vals + (size_t)slot * R + q * 4 * G + sub * 4) =
        zero ? make_float4(0.f, 0.f, 0.f, 0.f)
             : make_float4(acc[q * 4], acc[q * 4 + 1], acc[q * 4 + 2], acc[q * 4 + 3]);
}

template <int R, int V, int G>
__device__ __forceinline__ void det_plain(float* out, uint32_t row, int sub, const float (&acc)[V]) {
#pragma unroll
  for (int q = 0; q < V / 4; ++q) {
    float4* o = reinterpret_cast<float4*>(out + (size_t)row * R + q * 4 * G + sub * 4);
    float4 x = *o;
    x.x += acc[q * 4];
    x.y += acc[q * 4 + 1];
    x.z += acc[q * 4 + 2];
    x.w += acc[q * 4 + 3];
    *o = x;
  }
}

// The open run of a lane group (CARRY walks take it in and hand it back
// instead of updating the output at the end of their sub-range).
template <int V>
struct OpenRun {
  uint32_t row;
  float acc[V];
  // the deterministic walk's sum of the run so far, in pieces of kFoldSteps
  // steps: a run of n nonzeros is then a chain of n / kFoldSteps additions of
  // chains of kFoldSteps instead of one of n (5 modes, 5M nonzeros, rank 64: error
  // 1.4e-7 instead of 3.2e-7 for 2% of the time; the walk with atomics, whose
  // registers are all taken, lost 25% on the power-law 3-mode tensor)
  float sum[V];
  __device__ __forceinline__ void open() {
    row = 0xffffffffu;
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = sum[q] = 0.f;
  }
  __device__ __forceinline__ void fold() {
#pragma unroll
    for (int q = 0; q < V; ++q) {
      sum[q] += acc[q];
      acc[q] = 0.f;
    }
  }
  // acc: the whole run
  __device__ __forceinline__ void close() {
#pragma unroll
    for (int q = 0; q < V; ++q) {
      acc[q] += sum[q];
      sum[q] = 0.f;
    }
  }
};
constexpr uint32_t kFoldSteps = 16;

template <int R, typename FT, int HW, int NM, bool SMEM, bool DET = false, bool CARRY = false>
__device__ __forceinline__ void warp_range(const MttkrpArgs& a, const void* line, uint32_t ws, uint32_t we,
                                           bool staged, float* smem, uint32_t iv_start, uint32_t sr_base = 0,
                                           OpenRun<LaneWidth<R>::V>* carry = nullptr) {
  using LW = LaneWidth<R>;
  const int target = a.target;
  constexpr int V = LW::V, G = LW::G, NPW = LW::NPW;
  // nonzeros per step: 2 for 3 modes (4 measured faster for DET only), 1
  // beyond (two measured 30% slower on the rank-64 5-mode tensor: its four
  // gathered rows per nonzero already fill the registers); the accumulation
  // order is the line order whatever U is
  constexpr int U = NM <= 3 ? (DET ? 4 : 2) : 1;
  const int lane = threadIdx.x & 31;
  const int grp = lane / G, sub = lane % G;
  // groups' sub-ranges; odd lengths when reading shared memory, so the
  // groups' records fall in different banks
  uint32_t sublen = (we - ws + NPW - 1) / NPW;
  if (SMEM) sublen |= 1u;
  const uint32_t gs = min(ws + grp * sublen, we);
  const uint32_t ge = min(gs + sublen, we);
  float acc[V];
  uint32_t cur = kNoRow;
  if constexpr (CARRY) {
    cur = carry->row;
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = carry->acc[q];
  } else {
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = 0.f;
  }
  uint32_t nrun = 0;  // runs emitted (DET)
  const uint32_t slot0 = 2 * (sr_base + grp);

  uint32_t w[U][4];
  float v[U];
  bool valid[U];
  load_keys<HW, U, SMEM>(line, gs, ge, w, v, valid);
  for (uint32_t k = 0; k < sublen; k += U) {
    // factor rows of the NM-1 input modes (j-th input mode m = j, or j+1
    // past the target)
    float f[U][NM - 1][V];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < NM - 1; ++j) {
        const int m = j < target ? j : j + 1;
        if (m < a.dec.nmodes && valid[u]) {
          const uint32_t r = rec_row(w[u], a.dec, m);
          load_row<FT, V, G>(a.fac.f[m], (size_t)r * R, sub, f[u][j]);
        }
      }
    }
    uint32_t rows[U];
    float vals[U];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rows[u] = rec_row(w[u], a.dec, target);
      vals[u] = v[u];
      ok[u] = valid[u];
    }
    load_keys<HW, U, SMEM>(line, gs + k + U, ge, w, v, valid);  // next iteration's keys
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!ok[u]) continue;
      if constexpr (NM <= 5) {
        // exact mode count: packed FP32x2 products, the last factor fused
        // into the running sum (acc = p f_last, or acc += p f_last)
        float2 p2[V / 2];
#pragma unroll
        for (int h = 0; h < V / 2; ++h) {
          p2[h] = __fmul2_rn(make_float2(vals[u], vals[u]), make_float2(f[u][0][2 * h], f[u][0][2 * h + 1]));
#pragma unroll
          for (int j = 1; j < NM - 2; ++j)
            p2[h] = __fmul2_rn(p2[h], make_float2(f[u][j][2 * h], f[u][j][2 * h + 1]));
        }
        if (rows[u] != cur) {
          if (cur != kNoRow) {
            if (!DET)
              flush_row<R, V, G>(staged, smem, iv_start, a.out, cur, sub, acc);
            else if (nrun++ == 0)
              det_slot<R, V, G>(a, slot0, cur, sub, acc, false);
            else
              det_plain<R, V, G>(a.out, cur, sub, acc);
          }
          cur = rows[u];
#pragma unroll
          for (int h = 0; h < V / 2; ++h) {
            const float2 r2 = __fmul2_rn(p2[h], make_float2(f[u][NM - 2][2 * h], f[u][NM - 2][2 * h + 1]));
            acc[2 * h] = r2.x;
            acc[2 * h + 1] = r2.y;
          }
        } else {
#pragma unroll
          for (int h = 0; h < V / 2; ++h) {
            const float2 r2 = __ffma2_rn(p2[h], make_float2(f[u][NM - 2][2 * h], f[u][NM - 2][2 * h + 1]),
                                         make_float2(acc[2 * h], acc[2 * h + 1]));
            acc[2 * h] = r2.x;
            acc[2 * h + 1] = r2.y;
          }
        }
      } else {
        float p[V];
#pragma unroll
        for (int q = 0; q < V; ++q) p[q] = vals[u];
#pragma unroll
        for (int j = 0; j < NM - 1; ++j)
          if ((j < a.target ? j : j + 1) < a.dec.nmodes)
#pragma unroll
            for (int q = 0; q < V; ++q) p[q] *= f[u][j][q];
        if (rows[u] != cur) {
          if (cur != kNoRow) {
            if (!DET)
              flush_row<R, V, G>(staged, smem, iv_start, a.out, cur, sub, acc);
            else if (nrun++ == 0)
              det_slot<R, V, G>(a, slot0, cur, sub, acc, false);
            else
              det_plain<R, V, G>(a.out, cur, sub, acc);
          }
          cur = rows[u];
#pragma unroll
          for (int q = 0; q < V; ++q) acc[q] = p[q];
        } else {
#pragma unroll
          for (int q = 0; q < V; ++q) acc[q] += p[q];
        }
      }
    }
  }
  if (!DET) {
    if constexpr (CARRY) {
      carry->row = cur;
#pragma unroll
      for (int q = 0; q < V; ++q) carry->acc[q] = acc[q];
    } else if (cur != kNoRow) {
      flush_row<R, V, G>(staged, smem, iv_start, a.out, cur, sub, acc);
    }
  } else if (cur == kNoRow) {
    // empty sub-range: both slots carry the row of the entry before it (the
    // last run of an earlier sub-range) with zeros, keeping slot rows sorted
    uint32_t w0[1][4];
    float v0[1];
    bool ok0[1];
    const uint32_t at = gs > 0 ? gs - 1 : 0;
    load_keys<HW, 1, SMEM>(line, at, at + 1, w0, v0, ok0);
    const uint32_t r0 = rec_row(w0[0], a.dec, a.target);
    det_slot<R, V, G>(a, slot0, r0, sub, acc, true);
    det_slot<R, V, G>(a, slot0 + 1, r0, sub, acc, true);
  } else if (nrun == 0) {
    det_slot<R, V, G>(a, slot0, cur, sub, acc, false);
    det_slot<R, V, G>(a, slot0 + 1, cur, sub, acc, true);
  } else {
    det_slot<R, V, G>(a, slot0 + 1, cur, sub, acc, false);
  }
}

template <int R, typename FT, int HW, bool STAGE, int NM, bool DET = false>
__global__ void __launch_bounds__(kMttkrpThreads, 3)
    mttkrp_tile_kernel(const MttkrpArgs a) {
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int warp = threadIdx.x >> 5;
  const int N = a.dec.nmodes;
  if constexpr (!STAGE && !DET) {
    // chunks of chunk_tiles consecutive tiles, round robin over the blocks;
    // within a chunk each lane group walks its sub-range of every tile with
    // its open run carried along, so a row running through the chunk (a hot
    // row) is updated once per group and chunk rather than once per tile:
    // fewer float32 additions in the output, and fewer atomics
    using LW = LaneWidth<R>;
    const uint32_t ct = a.chunk_tiles ? a.chunk_tiles : 1;
    const uint32_t nchunks = (a.ntiles + ct - 1) / ct;
    for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
      OpenRun<LW::V> run;
      run.row = kNoRow;
#pragma unroll
      for (int q = 0; q < LW::V; ++q) run.acc[q] = 0.f;
      const uint32_t t_end = min(c * ct + ct, a.ntiles);
      for (uint32_t tile = c * ct; tile < t_end; ++tile) {
        const uint32_t ts = tile * a.tile_nnz;
        const uint32_t te = min(ts + a.tile_nnz, a.nnz);
        const uint32_t chunk = (te - ts + kMttkrpWarps - 1) / kMttkrpWarps;
        const uint32_t ws = min(ts + warp * chunk, te);
        const uint32_t we = min(ws + chunk, te);
        warp_range<R, FT, HW, NM, false, false, true>(a, a.line, ws, we, false, smem, 0, 0, &run);
      }
      if (run.row != kNoRow)
        flush_row<R, LW::V, LW::G>(false, smem, 0, a.out, run.row, (threadIdx.x & 31) % LW::G, run.acc);
    }
    return;
  }
  for (uint32_t tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
    const uint32_t ts = tile * a.tile_nnz;
    const uint32_t te = min(ts + a.tile_nnz, a.nnz);
    uint32_t iv_start = 0;
    bool staged = false;
    if (STAGE) {
      iv_start = a.tile_iv[((size_t)tile * N + a.target) * 2];
      const uint32_t iv_len = a.tile_iv[((size_t)tile * N + a.target) * 2 + 1];
      staged = iv_len <= (uint32_t)a.stage_rows && iv_len * 2 <= (te - ts);
      if (staged) {
        for (uint32_t q = threadIdx.x; q < iv_len * (R / 4); q += blockDim.x)
          smem4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
    }
    const uint32_t chunk = (te - ts + kMttkrpWarps - 1) / kMttkrpWarps;
    const uint32_t ws = min(ts + warp * chunk, te);
    const uint32_t we = min(ws + chunk, te);
    warp_range<R, FT, HW, NM, false, DET>(a, a.line, ws, we, staged, smem, iv_start,
                                          (tile * kMttkrpWarps + warp) * LaneWidth<R>::NPW);
    if (STAGE && staged) {
      __syncthreads();
      const uint32_t iv_len = a.tile_iv[((size_t)tile * N + a.target) * 2 + 1];
      for (uint32_t q = threadIdx.x; q < iv_len * (R / 4); q += blockDim.x) {
        const float4 v = smem4[q];
        if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f) {
          const uint32_t r = q / (R / 4), s = q % (R / 4);
          atomicAdd(reinterpret_cast<float4*>(a.out + (size_t)(iv_start + r) * R + s * 4), v);
        }
      }
      __syncthreads();
    }
  }
}

// ------------------------------------------------ the row-sorted walk
//
// SORTED and DETERMINISTIC on 3- to 5-mode tensors: the walk over a kDecoded
// copy.  As warp_range, a warp's range is split into NPW contiguous
// sub-ranges, one per lane group of G = R / V lanes; each lane holds V floats
// of every row.  A walk over the line's keys with four floats a lane was bound by
// issue slots (5 modes at rank 64: 64 warp instructions per nonzero), so a step
// does as little as possible besides its row loads: the rows come decoded, target
// last (no decode, no selection among the modes), the loads past the end of a
// sub-range are clamped to the last record instead of being predicated, and V is as
// wide as the registers allow, which divides the per-nonzero overhead by the
// nonzeros in flight.  Now the latency of the gathers bounds it (20 to 22
// instructions there, issue slots 33% busy in float32 and 55% in bfloat16, L1 66% and
// 58%; long walks of 3 modes 8.5 instructions and 40%).

template <int NIN>
struct DecRec {
  uint32_t in[NIN];
  uint32_t row;
  float v;
};

template <int NIN>
__device__ __forceinline__ DecRec<NIN> load_dec(const void* line, const void* extra, uint32_t i) {
  const uint4 q = __ldg(static_cast<const uint4*>(line) + i);
  DecRec<NIN> r;
  r.in[0] = q.x;
  r.in[1] = q.y;
  if constexpr (NIN == 2) {
    r.row = q.z;
    r.v = __uint_as_float(q.w);
  } else if constexpr (NIN == 3) {
    r.in[2] = q.z;
    r.row = q.w;
    r.v = __ldg(static_cast<const float*>(extra) + i);
  } else {
    r.in[2] = q.z;
    r.in[3] = q.w;
    const uint2 e = __ldg(static_cast<const uint2*>(extra) + i);
    r.row = e.x;
    r.v = __uint_as_float(e.y);
  }
  return r;
}

// How a lane group of the walk covers a row of R factors: V floats a lane in
// pieces of P floats (one load each: 16 bytes, or 8 for four bfloat16), piece
// p of lane `sub` at column p P G + P sub, so one load of the group's lanes
// reads P G consecutive factors.
template <int R, typename FT, int V>
struct WalkMap {
  static constexpr int G = R / V;
  static constexpr int NPW = 32 / G;
  static constexpr int P = sizeof(FT) == 4 ? 4 : (V < 8 ? V : 8);
  __device__ static int col(int q, int sub) {  // column of this lane's float4 q (q < V / 4)
    constexpr int H = P / 4;                   // float4s per piece
    return (q / H) * P * G + P * sub + (q % H) * 4;
  }
};

template <int R, typename FT, int V>
__device__ __forceinline__ void walk_row(const void* base, uint32_t row, int sub, float (&x)[V]) {
  using WM = WalkMap<R, FT, V>;
  const char* p = static_cast<const char*>(base) + (size_t)row * (R * sizeof(FT)) + (WM::P * sub) * sizeof(FT);
  if constexpr (sizeof(FT) == 4) {
#pragma unroll
    for (int q = 0; q < V / 4; ++q) {
      const float4 f = __ldg(reinterpret_cast<const float4*>(p + (size_t)q * WM::P * WM::G * sizeof(FT)));
      x[4 * q] = f.x;
      x[4 * q + 1] = f.y;
      x[4 * q + 2] = f.z;
      x[4 * q + 3] = f.w;
    }
  } else if constexpr (V >= 8) {
#pragma unroll
    for (int q = 0; q < V / 8; ++q) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(p + (size_t)q * WM::P * WM::G * sizeof(FT)));
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        x[8 * q + 2 * h] = __uint_as_float(w[h] << 16);
        x[8 * q + 2 * h + 1] = __uint_as_float(w[h] & 0xffff0000u);
      }
    }
  } else {
    const float4 f = load4<FT>(p, 0);
    x[0] = f.x;
    x[1] = f.y;
    x[2] = f.z;
    x[3] = f.w;
  }
}

template <int R, typename FT, int V>
__device__ __forceinline__ void walk_flush(float* out, uint32_t row, int sub, const float (&acc)[V]) {
  float* o = out + (size_t)row * R;
#pragma unroll
  for (int q = 0; q < V / 4; ++q)
    atomicAdd(reinterpret_cast<float4*>(o + WalkMap<R, FT, V>::col(q, sub)),
              make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]));
}

// The row pieces of U nonzeros in flight.
template <int NIN, int V, int U>
struct WalkStage {
  float f[U][NIN][V];
  uint32_t row[U];
  float v[U];
};

// The deterministic walk's meeting place (shared memory): per lane group its
// first and last run (entries 2 g and 2 g + 1; row kNoRow: none), per warp
// whether it is one run (then summed into its first entry), and the block's
// open run from tile to tile.
template <int R, int NPW>
struct DetTile {
  static constexpr int E = 2 * kMttkrpWarps * NPW;
  static constexpr int Q = R / 4;
  float4 val[E][Q];
  float4 carry[2][Q];
  uint32_t row[E];
  uint32_t carry_row[2];
  int one[kMttkrpWarps];
};

template <int R, int V, int G, int NPW>
__device__ __forceinline__ void det_entry(DetTile<R, NPW>& d, int e, uint32_t row, int sub, const float (&acc)[V]) {
  if (sub == 0) d.row[e] = row;
#pragma unroll
  for (int q = 0; q < V / 4; ++q)
    d.val[e][q * G + sub] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
}

__device__ __forceinline__ void add4(float4& x, const float4& y) {
  x.x += y.x;
  x.y += y.y;
  x.z += y.z;
  x.w += y.w;
}

// A finished run of the deterministic walk that is its row's only one.
__device__ __forceinline__ void det_put(const MttkrpArgs& a, float4* o, float4 x) {
  if (a.det_add) add4(x, *o);
  *o = x;
}

// Sub-range [gs, ge) of a lane group, `steps` steps of U nonzeros (the same
// for every group of the warp).  D steps are in the air: the rows of step
// k + D - 1 are requested, and the records of step k + 2 D - 1, before step k
// is summed.  The open run is taken from and left in `run`.  det (the
// deterministic walk): the first run to end goes to entry `ent` of it, the others
// straight to the output, whose rows they have to themselves; returns how many
// ended.
template <int R, typename FT, int NIN, int V, int U, int D, bool DET>
__device__ __forceinline__ uint32_t walk_range(const MttkrpArgs& a, uint32_t gs, uint32_t ge, uint32_t steps, int sub,
                                               OpenRun<V>& run,
                                               DetTile<R, WalkMap<R, FT, V>::NPW>* det = nullptr, int ent = 0) {
  const void* base[NIN];
#pragma unroll
  for (int j = 0; j < NIN; ++j) base[j] = a.in.f[j];
  const void* line = a.line;
  const void* extra = a.extra;
  const uint32_t last = a.nnz - 1;
  uint32_t nrun = 0;
  DecRec<NIN> rec[D][U];
  WalkStage<NIN, V, U> st[D];
  auto fetch = [&](DecRec<NIN>(&r)[U], uint32_t at) {
#pragma unroll
    for (int u = 0; u < U; ++u) r[u] = load_dec<NIN>(line, extra, min(at + u, last));
  };
  auto issue = [&](WalkStage<NIN, V, U>& s, const DecRec<NIN>(&r)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int j = 0; j < NIN; ++j) walk_row<R, FT, V>(base[j], r[u].in[j], sub, s.f[u][j]);
      s.row[u] = r[u].row;
      s.v[u] = r[u].v;
    }
  };
  auto sum = [&](const WalkStage<NIN, V, U>& s, uint32_t at) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (at + u >= ge) continue;
      float2 p[V / 2];  // packed FP32x2, the last factor fused into the sum
#pragma unroll
      for (int h = 0; h < V / 2; ++h) {
        p[h] = __fmul2_rn(make_float2(s.v[u], s.v[u]), make_float2(s.f[u][0][2 * h], s.f[u][0][2 * h + 1]));
#pragma unroll
        for (int j = 1; j < NIN - 1; ++j)
          p[h] = __fmul2_rn(p[h], make_float2(s.f[u][j][2 * h], s.f[u][j][2 * h + 1]));
      }
      if (s.row[u] != run.row) {
        if (run.row != kNoRow) {
          if constexpr (DET) run.close();
          if constexpr (!DET) {
            walk_flush<R, FT, V>(a.out, run.row, sub, run.acc);
          } else {
            constexpr int G = WalkMap<R, FT, V>::G;
            if (nrun++ == 0) {
              det_entry<R, V, G>(*det, ent, run.row, sub, run.acc);
            } else {
#pragma unroll
              for (int q = 0; q < V / 4; ++q)
                det_put(a, reinterpret_cast<float4*>(a.out + (size_t)run.row * R + WalkMap<R, FT, V>::col(q, sub)),
                        make_float4(run.acc[4 * q], run.acc[4 * q + 1], run.acc[4 * q + 2], run.acc[4 * q + 3]));
            }
          }
        }
        run.row = s.row[u];
#pragma unroll
        for (int h = 0; h < V / 2; ++h) {
          const float2 x = __fmul2_rn(p[h], make_float2(s.f[u][NIN - 1][2 * h], s.f[u][NIN - 1][2 * h + 1]));
          run.acc[2 * h] = x.x;
          run.acc[2 * h + 1] = x.y;
        }
      } else {
#pragma unroll
        for (int h = 0; h < V / 2; ++h) {
          const float2 x = __ffma2_rn(p[h], make_float2(s.f[u][NIN - 1][2 * h], s.f[u][NIN - 1][2 * h + 1]),
                                      make_float2(run.acc[2 * h], run.acc[2 * h + 1]));
          run.acc[2 * h] = x.x;
          run.acc[2 * h + 1] = x.y;
        }
      }
    }
  };
#pragma unroll
  for (int d = 0; d < D; ++d) fetch(rec[d], gs + d * U);
#pragma unroll
  for (int d = 0; d < D - 1; ++d) {
    issue(st[d], rec[d]);
    fetch(rec[d], gs + (d + D) * U);
  }
  uint32_t i = gs;
  for (uint32_t k = 0; k < steps; k += D, i += D * U) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      constexpr int kAhead = D - 1;
      issue(st[(d + kAhead) % D], rec[(d + kAhead) % D]);
      fetch(rec[(d + kAhead) % D], i + (d + kAhead + D) * U);
      sum(st[d], i + d * U);
    }
    if (DET && (k & (kFoldSteps - 1)) == kFoldSteps - D) run.fold();
  }
  return nrun;
}

// The widths of the walk: V floats a lane, U nonzeros a step, D steps in the
// air, MINB blocks an SM (the register budget), by rank, input modes and
// factor type.  Eight floats a lane halve the instructions per nonzero but
// also the lanes per nonzero, so there are twice as many lane groups, with
// runs half as long and twice the updates: measured better at rank 64 (5 modes,
// 12M nonzeros: float32 631 us against 645, bfloat16 494 against 541) and worse
// at rank 16 and 32 (power-law 3-mode, 40M nonzeros, rank 32: 936 us against
// 809; uniform 1000^3, 1M nonzeros, rank 16: 27.6 against 21.5).  3 modes in
// float32 wait for their rows (two loads a nonzero, the longest stall by far).
// Rows from L2 want the blocks: one step in the air at five blocks an SM took
// 3 to 15% less than two at three from 9M to 40M nonzeros at ranks 8, 16 and 32
// (uniform, rows of 15 to 32 MB, 25M: 264 us against 288 at rank 16, 443 against
// 474 at rank 32; 1000 rows, 40M, rank 16: 350 against 394; by at most 3% more,
// 15M at rank 8).  Rows from memory are better asked for two steps ahead, or
// as fast (40M distinct nonzeros over 4.8M x 1.8M x 1.8M, rank 32, three modes:
// 2433 us against 2508 at the same error; power law, 15M, rank 16: 201 against
// 223 and 213, but rank 8 121 against 118); with more rows per nonzero two steps
// spill (2.1 ms against 0.63).
template <int R, typename FT, int NIN, bool DET, bool DEEP = false>
struct WalkCfg {
  static constexpr int V = R >= 64 ? 8 : 4;
  static constexpr int U = V == 4 && (NIN == 2 || (NIN == 3 && DET)) ? 2 : 1;
  static constexpr int D = DEEP ? 2 : 1;
  static constexpr int MINB = DEEP ? 3 : NIN == 2 && V == 4 && !DET ? 5 : 4;
};
// Whether two steps in the air pay: 3 modes in float32 whose walk is long
// (kDeepNnz: 5M nonzeros 124 us against 119) and whose input factors are more
// than the L2 holds (launch_walk).
template <int R, typename FT, int NIN>
constexpr bool kCanBeDeep = NIN == 2 && R < 64 && sizeof(FT) == 4;
constexpr uint32_t kDeepNnz = 8u << 20;

// This lane's group's part of warp `warp`'s share of tile `tile`.
template <int NPW, int G, int U>
struct TilePart {
  uint32_t gs, ge, steps;
  __device__ TilePart(const MttkrpArgs& a, uint32_t tile, int warp, int grp) {
    const uint32_t ts = tile * a.tile_nnz;
    const uint32_t te = min(ts + a.tile_nnz, a.nnz);
    const uint32_t chunk = (te - ts + kMttkrpWarps - 1) / kMttkrpWarps;
    const uint32_t ws = min(ts + warp * chunk, te);
    const uint32_t we = min(ws + chunk, te);
    const uint32_t sublen = (we - ws + NPW - 1) / NPW;
    gs = min(ws + grp * sublen, we);
    ge = min(gs + sublen, we);
    steps = (sublen + U - 1) / U;
  }
};

// The lane groups' open runs at the end of a chunk: when a whole warp ends on
// one row (a hot row, or a mode of few rows) its groups are summed first, by a
// tree, and the row is updated once instead of once per group.  Groups
// of G lanes; lanes past the last group, and groups without records (the ragged
// end of a tile), hold zeros.
template <int V>
__device__ __forceinline__ bool merge_groups(uint32_t row, float (&acc)[V], int G, int npw, int lane) {
  const uint32_t row0 = __shfl_sync(0xffffffffu, row, 0);
  if (!__all_sync(0xffffffffu, row == row0 || row == kNoRow || lane >= G * npw)) return false;
  for (int live = npw, half; live > 1; live = half) {
    half = (live + 1) / 2;
#pragma unroll
    for (int q = 0; q < V; ++q) {
      const float x = __shfl_sync(0xffffffffu, acc[q], (lane + half * G) & 31);
      if (lane < (live - half) * G) acc[q] += x;
    }
  }
  return true;
}

template <int R, typename FT, int NIN, bool DEEP>
__global__ void __launch_bounds__(kMttkrpThreads, WalkCfg<R, FT, NIN, false, DEEP>::MINB)
    walk_kernel(const MttkrpArgs a) {
  using C = WalkCfg<R, FT, NIN, false, DEEP>;
  using WM = WalkMap<R, FT, C::V>;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / WM::G, sub = lane % WM::G;
  // chunks of consecutive tiles, the open run carried through them (as in
  // mttkrp_tile_kernel)
  const uint32_t ct = a.chunk_tiles ? a.chunk_tiles : 1;
  const uint32_t nchunks = (a.ntiles + ct - 1) / ct;
  for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
    OpenRun<C::V> run;
    run.open();
    const uint32_t t_end = min(c * ct + ct, a.ntiles);
    for (uint32_t tile = c * ct; tile < t_end; ++tile) {
      const TilePart<WM::NPW, WM::G, C::U> p(a, tile, warp, grp);
      walk_range<R, FT, NIN, C::V, C::U, C::D, false>(a, p.gs, p.ge, p.steps, sub, run);
    }
    const bool one = WM::NPW > 1 && merge_groups<C::V>(run.row, run.acc, WM::G, WM::NPW, lane);
    if (run.row != kNoRow && !(one && grp)) walk_flush<R, FT, C::V>(a.out, run.row, sub, run.acc);
  }
}

// Chunk `chunk` of the deterministic walk (one block): consecutive tiles, each
// cut among the lane groups as any walk's.  What a group starts and ends with
// meets in shared memory, where runs that cross groups are summed in a fixed
// order; the block's open run is carried from tile to tile, its first and last
// run go to the chunk's two slots (det_fix_kernel), and every other run is its
// row's only one and is written without atomics.  So the slots are two per
// block, however short the groups' sub-ranges are cut for latency: with two per
// sub-range, the slots of a 200,000-nonzero slice were half its nonzeros and their
// fix-up (three launches, 24 us) took longer than the walk (9 us).
template <int R, int NIN>
__device__ __forceinline__ void det_walk_chunk(const MttkrpArgs& a, uint32_t chunk) {
  using C = WalkCfg<R, float, NIN, true>;
  using WM = WalkMap<R, float, C::V>;
  using DT = DetTile<R, WM::NPW>;
  constexpr int E = DT::E, Q = DT::Q, kPerWarp = 2 * WM::NPW, kAhead = 4;
  __shared__ DT d;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / WM::G, sub = lane % WM::G;
  const uint32_t t0 = chunk * a.chunk_tiles, t1 = min(t0 + a.chunk_tiles, a.ntiles);
  const uint32_t first_row = load_dec<NIN>(a.line, a.extra, t0 * a.tile_nnz).row;
  const uint32_t slot = 2 * chunk;
  auto put = [&](uint32_t row, int q, float4 x) {  // a finished run of the block
    if (row == first_row)
      *reinterpret_cast<float4*>(a.det_vals + (size_t)slot * R + q * 4) = x;
    else
      det_put(a, reinterpret_cast<float4*>(a.out + (size_t)row * R + q * 4), x);
  };
  if (threadIdx.x == 0) d.carry_row[0] = kNoRow;
  int cur = 0;
  for (uint32_t tile = t0; tile < t1; ++tile) {
    const TilePart<WM::NPW, WM::G, C::U> p(a, tile, warp, grp);
    const int ent = 2 * (warp * WM::NPW + grp);
    OpenRun<C::V> run;
    run.open();
    const uint32_t ended = walk_range<R, float, NIN, C::V, C::U, C::D, true>(a, p.gs, p.ge, p.steps, sub, run, &d, ent);
    run.close();
    const bool one = __all_sync(0xffffffffu, ended == 0) &&
                     merge_groups<C::V>(run.row, run.acc, WM::G, WM::NPW, lane);
    if (lane == 0) d.one[warp] = one;
    if (run.row == kNoRow || (one && grp)) {
      if (sub == 0) d.row[ent] = d.row[ent + 1] = kNoRow;
    } else if (ended == 0) {
      det_entry<R, C::V, WM::G>(d, ent, run.row, sub, run.acc);
      if (sub == 0) d.row[ent + 1] = kNoRow;
    } else {
      det_entry<R, C::V, WM::G>(d, ent + 1, run.row, sub, run.acc);
    }
    __syncthreads();
    const uint32_t open = d.carry_row[cur];
    if (threadIdx.x < Q && open != kNoRow && open != d.row[0]) put(open, threadIdx.x, d.carry[cur][threadIdx.x]);
    for (int w = threadIdx.x; w < E * Q; w += kMttkrpThreads) {
      const int e = w / Q, q = w % Q;
      const uint32_t r = d.row[e];
      if (r == kNoRow) continue;
      int prev = e - 1;
      if (prev >= 0 && d.one[prev / kPerWarp]) prev -= prev % kPerWarp;  // (a merged warp's one entry is its first)
      while (prev >= 0 && d.row[prev] == kNoRow) --prev;
      if (prev >= 0 && d.row[prev] == r) continue;  // not the first entry of its run
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), upper = x, part = x;
      bool ends = false;
      // (a merged warp has one entry; of the others four are loaded at a time, or
      // each would wait for the one before it: 90 cycles an entry, 12 us for a
      // chunk of one row at rank 8.  The entries of a warp are summed in `part`, the
      // warps of each half of the block in x and `upper`: one after the other all
      // made the error of rows of some hundred nonzeros, 500 rows at rank 8 7.2e-8
      // rms from 50,000 nonzeros and 6.7e-8 from 1M, now 4.5e-8 both)
      for (int k = e; k < E && !ends;) {
        const bool merged = d.one[k / kPerWarp];
        const int stop = k - k % kPerWarp + kPerWarp;
        uint32_t rk[kAhead];
        float4 y[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const bool in = k + u < stop && (u == 0 || !merged);
          rk[u] = in ? d.row[k + u] : kNoRow;
          y[u] = d.val[min(k + u, E - 1)][q];
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (ends || rk[u] == kNoRow) continue;
          if (rk[u] != r) {
            ends = true;
            continue;
          }
          add4(part, y[u]);
        }
        k = merged ? stop : min(k + kAhead, stop);
        if (k == stop || ends) {
          if (k <= E / 2)
            add4(x, part);
          else
            add4(upper, part);
          part = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      add4(x, upper);
      if (prev < 0 && open == r) add4(x, d.carry[cur][q]);
      if (ends) {
        put(r, q, x);
      } else {
        d.carry[cur ^ 1][q] = x;
        if (q == 0) d.carry_row[cur ^ 1] = r;
      }
    }
    __syncthreads();
    cur ^= 1;
  }
  // the open run: the chunk's last slot, or its first if that is still the same run
  const uint32_t row = d.carry_row[cur];
  if (threadIdx.x < Q) {
    const float4 x = d.carry[cur][threadIdx.x];
    const bool single = row == first_row;
    float4* s = reinterpret_cast<float4*>(a.det_vals + (size_t)slot * R) + threadIdx.x;
    if (single) s[0] = x;
    s[Q] = single ? make_float4(0.f, 0.f, 0.f, 0.f) : x;
    if (threadIdx.x == 0) {
      a.det_rows[slot] = first_row;
      a.det_rows[slot + 1] = row;
    }
  }
  __syncthreads();
}

template <int R, int NIN>
__global__ void __launch_bounds__(kMttkrpThreads, 3) det_walk_kernel(const MttkrpArgs a) {
  det_walk_chunk<R, NIN>(a, blockIdx.x);
}

// The chunks' slots (rows non-decreasing; a row in them is in no other run):
// a block per run of equal rows, its slots summed in float64 with a fixed split
// and a fixed tree, then written or added to the row (60 rows at rank 8 from 1M
// nonzeros: 4.9e-8 rms error with float32 sums, 3.1e-8 so, in the same time).
// What it waits for is one SM's loads of a single row's slots (780 at rank 64:
// 15 us with the loads one after the other, 8.9 us with eight in the air); 3 us when
// every row has a few slots.  Block `first` of `step` that share the item.
struct __align__(16) Sum4 {
  double x, y, z, w;
};
__device__ __forceinline__ void det_fix_slots(const MttkrpArgs& a, uint32_t nslots, int R, Sum4* part,
                                              uint32_t first, uint32_t step) {
  const uint32_t* rows = a.det_rows;
  const float4* vals = reinterpret_cast<const float4*>(a.det_vals);
  const int Q = R / 4, S = 256 / Q;
  const int s = threadIdx.x / Q, q = threadIdx.x % Q;
  for (uint32_t i = first; i < nslots; i += step) {
    const uint32_t row = rows[i];
    if (i > 0 && rows[i - 1] == row) continue;
    uint32_t end = i + 1;
    for (;;) {  // (the rows are sorted: the equal ones of a window of 1024 come first)
      uint32_t next[4];
#pragma unroll
      for (uint32_t u = 0; u < 4; ++u) {
        const uint32_t k = end + u * 256 + threadIdx.x;
        next[u] = k < nslots ? rows[k] : ~row;
      }
      int same = 0;
#pragma unroll
      for (int u = 0; u < 4; ++u) same += __syncthreads_count(next[u] == row);
      end += same;
      if (same < 1024) break;
    }
    Sum4 x = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t k = i + s; k < end; k += 8 * S) {  // (eight loads in the air)
      float4 y[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        y[u] = k + u * S < end ? vals[(size_t)(k + u * S) * Q + q] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int stride = 4; stride >= 1; stride >>= 1)
#pragma unroll
        for (int u = 0; u < stride; ++u) add4(y[u], y[u + stride]);
      x.x += y[0].x;
      x.y += y[0].y;
      x.z += y[0].z;
      x.w += y[0].w;
    }
    part[threadIdx.x] = x;
    __syncthreads();
    int live = S;
    while (live > 1 && live / 2 >= (int)(end - i)) live /= 2;  // (the rest are zeros)
    for (int stride = live / 2; stride >= 1; stride >>= 1) {
      if (s < stride) {
        const Sum4 y = part[(s + stride) * Q + q];
        Sum4& m = part[s * Q + q];
        m.x += y.x;
        m.y += y.y;
        m.z += y.z;
        m.w += y.w;
      }
      __syncthreads();
    }
    if (s == 0) {
      const Sum4 t = part[q];
      det_put(a, reinterpret_cast<float4*>(a.out + (size_t)row * R) + q,
              make_float4((float)t.x, (float)t.y, (float)t.z, (float)t.w));
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) det_fix_kernel(const MttkrpArgs a, uint32_t nslots, int R) {
  __shared__ Sum4 part[256];
  det_fix_slots(a, nslots, R, part, blockIdx.x, gridDim.x);
}

// ------------------------------------------------ deterministic fix-up
//
// (Lines that are not decoded: 2 modes, or more than 5.)  The slots of DET hold,
// in line order, the first and last run of every sub-range; their rows are non-decreasing, and a row appears in the slots
// only if it is in none of the interior runs.  A chain (maximal stretch of
// slots with one row) is summed in slot order, by one warp when it is short
// and by one block with a fixed split and a fixed tree when it is long (a
// hot row, or the single row of the stream mode).  The summation order is a
// function of nnz, the rank and the line alone, so results repeat bit for
// bit from run to run and whatever else runs on the device.

constexpr uint32_t kShortChain = 64;
constexpr uint32_t kChainSeg = 256;  // slots per segment of a long chain

// Chain starting at slot i (one warp; lanes cooperate): a short chain is
// summed in slot order into its row; a long one registers itself and its
// segments for det_fix_seg / det_fix_final.
__device__ __forceinline__ void det_short_chain(const uint32_t* __restrict__ rows, const float* __restrict__ vals,
                                                uint32_t nslots, int R, float* __restrict__ out, const DetLong& dl,
                                                uint32_t i, int lane) {
  const uint32_t row = rows[i];
  if (i > 0 && rows[i - 1] == row) return;  // not the head of its chain
  // chain end: first slot with a larger row -- the next 32 slots in one
  // coalesced probe, a binary search beyond them
  const uint32_t pi = i + 1 + lane;
  const unsigned differ = __ballot_sync(0xffffffffu, pi < nslots && rows[pi] != row);
  uint32_t lo;
  if (differ) {
    lo = i + 1 + __ffs(differ) - 1;
  } else if (i + 33 >= nslots) {
    lo = nslots;
  } else {
    lo = i + 33;
    uint32_t hi = nslots;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (rows[mid] == row)
        lo = mid + 1;
      else
        hi = mid;
    }
  }
  if (lo - i > kShortChain) {
    // long chain: register it and its segments (the order of the lists
    // varies from run to run; what each entry sums does not)
    const uint32_t nseg = (lo - i + kChainSeg - 1) / kChainSeg;
    uint32_t c = 0, base = 0;
    if (lane == 0) {
      c = atomicAdd(&dl.counters[0], 1u);
      base = atomicAdd(&dl.counters[1], nseg);
      dl.chains[c] = make_uint4(i, lo, base, nseg);
    }
    c = __shfl_sync(0xffffffffu, c, 0);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (uint32_t k = lane; k < nseg; k += 32) dl.segs[base + k] = make_uint2(c, k);
    return;
  }
  for (int r = lane; r < R; r += 32) {
    float x = 0.f;
    for (uint32_t k = i; k < lo; ++k) x += vals[(size_t)k * R + r];
    out[(size_t)row * R + r] += x;
  }
}

__global__ void __launch_bounds__(256)
    det_fix_short_kernel(const uint32_t* __restrict__ rows, const float* __restrict__ vals, uint32_t nslots,
                         int R, float* __restrict__ out, DetLong dl) {
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = gw; i < nslots; i += nw) det_short_chain(rows, vals, nslots, R, out, dl, i, lane);
}

// One segment g of a long chain (one block): thread (s, q) sums slots
// start+s, start+s+S, ... of rank quad q (S = 256 / (R/4)), then a fixed tree
// over s; the segment's R sums go to segpart.
__device__ __forceinline__ void det_segment(const float* __restrict__ vals, int R, const DetLong& dl, uint32_t g,
                                            float4* part) {
  const int Q = R / 4, S = 256 / Q;
  const int sidx = threadIdx.x / Q, q = threadIdx.x % Q;
  const uint2 sg = dl.segs[g];
  const uint4 ch = dl.chains[sg.x];
  const uint32_t s0 = ch.x + sg.y * kChainSeg;
  const uint32_t s1 = min(s0 + kChainSeg, ch.y);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (sidx < S)
    for (uint32_t k = s0 + sidx; k < s1; k += S) {
      const float4 v = *reinterpret_cast<const float4*>(vals + (size_t)k * R + q * 4);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int stride = S / 2; stride >= 1; stride >>= 1) {
    if (sidx < stride) {
      const float4 o = part[(sidx + stride) * Q + q];
      float4& m = part[sidx * Q + q];
      m.x += o.x;
      m.y += o.y;
      m.z += o.z;
      m.w += o.w;
    }
    __syncthreads();
  }
  if (sidx == 0) *reinterpret_cast<float4*>(dl.segpart + (size_t)(ch.z + sg.y) * R + q * 4) = part[q];
  __syncthreads();
}

__global__ void __launch_bounds__(256)
    det_fix_seg_kernel(const float* __restrict__ vals, int R, DetLong dl) {
  __shared__ float4 part[256];
  const uint32_t nseg = dl.counters[1];
  for (uint32_t g = blockIdx.x; g < nseg; g += gridDim.x) det_segment(vals, R, dl, g, part);
}

// One long chain c (one block): thread (s, q) sums segments s, s+S, ... of
// rank quad q, then a fixed tree over s; the result is added to the chain's
// row.
__device__ __forceinline__ void det_chain_final(const uint32_t* __restrict__ rows, int R, float* __restrict__ out,
                                                const DetLong& dl, uint32_t c, float4* part) {
  const int Q = R / 4, S = 256 / Q;
  const int sidx = threadIdx.x / Q, q = threadIdx.x % Q;
  const uint4 ch = dl.chains[c];
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (sidx < S)
    for (uint32_t k = sidx; k < ch.w; k += S) {
      const float4 v = *reinterpret_cast<const float4*>(dl.segpart + (size_t)(ch.z + k) * R + q * 4);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int stride = S / 2; stride >= 1; stride >>= 1) {
    if (sidx < stride) {
      const float4 o = part[(sidx + stride) * Q + q];
      float4& m = part[sidx * Q + q];
      m.x += o.x;
      m.y += o.y;
      m.z += o.z;
      m.w += o.w;
    }
    __syncthreads();
  }
  if (sidx == 0) {
    float4* o = reinterpret_cast<float4*>(out + (size_t)rows[ch.x] * R + q * 4);
    float4 x = *o;
    const float4 p = part[q];
    x.x += p.x;
    x.y += p.y;
    x.z += p.z;
    x.w += p.w;
    *o = x;
  }
  __syncthreads();
}

// The long-chain count of dl (every thread of the block gets it); the last
// block to have read it clears the counters for the next call (they start
// at zero when the workspace is allocated).
__device__ __forceinline__ uint32_t det_take_chains(const DetLong& dl, uint32_t* s_nlong) {
  if (threadIdx.x == 0) *s_nlong = dl.counters[0];
  __syncthreads();
  const uint32_t nlong = *s_nlong;
  if (threadIdx.x == 0 && atomicAdd(&dl.counters[2], 1u) == gridDim.x - 1) {
    dl.counters[0] = 0;
    dl.counters[1] = 0;
    dl.counters[2] = 0;
  }
  __syncthreads();
  return nlong;
}

__global__ void __launch_bounds__(256)
    det_fix_final_kernel(const uint32_t* __restrict__ rows, int R, float* __restrict__ out, DetLong dl) {
  __shared__ float4 part[256];
  __shared__ uint32_t s_nlong;
  const uint32_t nlong = det_take_chains(dl, &s_nlong);
  for (uint32_t c = blockIdx.x; c < nlong; c += gridDim.x) det_chain_final(rows, R, out, dl, c, part);
}

// ------------------------------------------------ grouped deterministic MTTKRP
//
// The same kernels over a table of items (sessions' MTTKRPs, one mode each):
// a global tile index runs over the items' tiles (prefix sums tile_off), and
// the fix-ups walk every item's slots, segments and chains in turn.  An
// item's sums, and their order, are those of its own launch.

__device__ __forceinline__ bool item_live(const int* active) { return !active || *active; }

// The last s in [0, K) with off[s] <= v (items with no blocks are skipped).
__device__ __forceinline__ int item_of(const uint32_t* __restrict__ off, int K, uint32_t v) {
  int lo = 0, hi = K;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// A grid's blocks split evenly among the items (several items per block when
// there are more items than blocks): every block going through all the items is
// a chain of dependent loads per item (the fix-up of four served slices of
// 50,000 nonzeros: 11.4 us so, 7.1 us split).
struct ItemShare {
  uint32_t items, blocks;        // items; blocks per item
  uint32_t item, block, stride;  // this block's first item, its place there, items between its items
  __device__ __forceinline__ explicit ItemShare(int count) {
    items = count > 0 ? (uint32_t)count : 0;
    blocks = items ? max(gridDim.x / items, 1u) : 1;
    stride = max(gridDim.x / blocks, 1u);
    item = blockIdx.x / blocks;
    block = blockIdx.x % blocks;
    if (item >= stride) item = items;  // (the remainder of the split)
  }
};

__global__ void __launch_bounds__(256) det_zero_group_kernel(Strided<DetItem> items) {
  const ItemShare sh(*items.count);
  const uint64_t tid = sh.block * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t nth = (uint64_t)sh.blocks * blockDim.x;
  for (uint32_t s = sh.item; s < sh.items; s += sh.stride) {
    const DetItem& it = items[s];
    if (!item_live(it.active)) continue;
    float4* o = reinterpret_cast<float4*>(it.a.out);
    const uint64_t n4 = it.out_floats / 4;
    for (uint64_t q = tid; q < n4; q += nth) o[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

template <int R, int NIN>
__global__ void __launch_bounds__(kMttkrpThreads, 3)
    det_tile_group_kernel(Strided<DetItem> items, const uint32_t* __restrict__ tile_off) {
  // the item's arguments staged in shared memory: the walk reads them per
  // nonzero (as a launch of its own reads them from the parameter bank)
  __shared__ MttkrpArgs sa;
  __shared__ int s_item;
  const int K = *items.count;
  const uint32_t total = K > 0 ? tile_off[K] : 0;
  if (threadIdx.x == 0) s_item = -1;
  for (uint32_t v = blockIdx.x; v < total; v += gridDim.x) {
    const int s = item_of(tile_off, K, v);
    const DetItem& it = items[s];
    if (!item_live(it.active)) continue;
    __syncthreads();  // (everyone is done with the previous item's copy)
    if (s != s_item) {
      constexpr int kWords = (int)(sizeof(MttkrpArgs) / 4);
      const uint32_t* src = reinterpret_cast<const uint32_t*>(&it.a);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&sa);
      for (int q = threadIdx.x; q < kWords; q += blockDim.x) dst[q] = src[q];
      __syncthreads();
      if (threadIdx.x == 0) s_item = s;
    }
    __syncthreads();
    det_walk_chunk<R, NIN>(sa, v - tile_off[s]);
  }
}

__global__ void __launch_bounds__(256) det_fix_group_kernel(Strided<DetItem> items, int R) {
  __shared__ Sum4 part[256];
  const ItemShare sh(*items.count);
  for (uint32_t s = sh.item; s < sh.items; s += sh.stride) {
    const DetItem& it = items[s];
    if (!item_live(it.active)) continue;
    det_fix_slots(it.a, it.nslots, R, part, sh.block, sh.blocks);
  }
}

// ------------------------------------------- line tiles staged by bulk copy
//
// The non-staged variants (ATOMIC, SORTED) stream the line through shared
// memory: per CTA, tiles of kLineTile entries are copied global -> shared by
// the bulk-copy engine (cp.async.bulk, completion on an mbarrier), double
// buffered, so the next tile is in flight while this one is walked.  The
// keys then come from shared memory (broadcast reads) and the LSU pipe
// carries only the factor-row gathers.  Waits are bounded: a wait that runs
// out sets *err and the whole block leaves after a second bounded wait for
// its copies in flight.

constexpr uint32_t kLineTile = 1024;
constexpr uint32_t kSpinLimit = 1u << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t phase) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t phase) {
  for (uint32_t spin = 0; spin < kSpinLimit; ++spin)
    if (mbar_try_wait(bar, phase)) return true;
  return false;
}

template <int R, typename FT, int HW, int NM>
__global__ void __launch_bounds__(kMttkrpThreads, 3)
    mttkrp_tma_kernel(const MttkrpArgs a, int* __restrict__ err) {
  constexpr uint32_t kRec = HW == 2 ? 32 : 16;  // record bytes
  constexpr uint32_t kBuf = kLineTile * kRec;
  extern __shared__ __align__(128) unsigned char sline[];
  __shared__ __align__(8) uint64_t bars[2];
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t ntiles = (a.nnz + kLineTile - 1) / kLineTile;

  auto buf = [&](int b) { return static_cast<void*>(sline + b * kBuf); };
  auto issue = [&](uint32_t tile, int b) {
    const uint32_t s0 = tile * kLineTile;
    const uint32_t n = min(kLineTile, a.nnz - s0);
    mbar_expect_tx(&bars[b], n * kRec);
    bulk_g2s(buf(b), static_cast<const unsigned char*>(a.line) + (size_t)s0 * kRec, n * kRec, &bars[b]);
  };

  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    if (blockIdx.x < ntiles) issue(blockIdx.x, 0);
    if (blockIdx.x + gridDim.x < ntiles) issue(blockIdx.x + gridDim.x, 1);
  }
  uint32_t it = 0;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
    const int b = it & 1;
    const uint32_t phase = (it >> 1) & 1;
    const bool ok = mbar_wait_bounded(&bars[b], phase);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicExch(err, 1);
        // the other buffer may still have a copy in flight: give it a bounded wait
        mbar_wait_bounded(&bars[b ^ 1], ((it + 1) >> 1) & 1);
      }
      return;
    }
    const uint32_t s0 = tile * kLineTile;
    const uint32_t n = min(kLineTile, a.nnz - s0);
    const uint32_t chunk = (n + kMttkrpWarps - 1) / kMttkrpWarps;
    const uint32_t ws = min(warp * chunk, n);
    const uint32_t we = min(ws + chunk, n);
    warp_range<R, FT, HW, NM, true>(a, buf(b), ws, we, false, nullptr, 0);
    __syncthreads();  // every warp is done with buffer b
    if (tid == 0) {
      const uint32_t nt = tile + 2 * gridDim.x;
      if (nt < ntiles) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(nt, b);
      }
    }
  }
}

// ------------------------------------------------ any rank, any alignment
//
// The walk at a rank (or alignment) the specialised kernels do not take: a
// lane group of G = ceil(R / V) lanes per nonzero -- any G up to 32, so 32 / G
// groups share a warp -- each lane holding V = 4 factors in V / VW loads of VW
// factors, VW the widest of 4, 2, 1 that divides the rank and that every
// pointer is aligned for.  Sub-ranges, runs and chunks are the specialised
// walk's (one vector atomic per run and lane); ranks above 128 take one
// column window of 128 per blockIdx.y.  Bound by the L1's load path (rank 10 over a
// row-sorted copy: 91% busy, 72 us for 3M nonzeros of a ragged 4-mode tensor) and,
// where runs are short, by atomics.  A warp per nonzero with a scalar atomic per
// factor, its form before, took 802 us there, at any of the line orders.
// STAGE: the runs of a line's mode of few rows are added in shared memory first
// (launch_any).

template <typename FT, int VW>
__device__ __forceinline__ void any_piece(const char* p, float* x) {
  if constexpr (VW == 4) {
    const float4 f = load4<FT>(p, 0);
    x[0] = f.x;
    x[1] = f.y;
    x[2] = f.z;
    x[3] = f.w;
  } else if constexpr (sizeof(FT) == 4) {
    if constexpr (VW == 2) {
      const float2 f = __ldg(reinterpret_cast<const float2*>(p));
      x[0] = f.x;
      x[1] = f.y;
    } else {
      x[0] = __ldg(reinterpret_cast<const float*>(p));
    }
  } else if constexpr (VW == 2) {
    const uint32_t u = __ldg(reinterpret_cast<const uint32_t*>(p));
    x[0] = __uint_as_float(u << 16);
    x[1] = __uint_as_float(u & 0xffff0000u);
  } else {
    x[0] = __uint_as_float((uint32_t)__ldg(reinterpret_cast<const unsigned short*>(p)) << 16);
  }
}

template <int VW>
__device__ __forceinline__ void any_flush(float* o, const float* x) {
  if constexpr (VW == 4)
    atomicAdd(reinterpret_cast<float4*>(o), make_float4(x[0], x[1], x[2], x[3]));
  else if constexpr (VW == 2)
    atomicAdd(reinterpret_cast<float2*>(o), make_float2(x[0], x[1]));
  else
    atomicAdd(o, x[0]);
}

// A record of either kind: DEC reads a kDecoded copy of NIN + 1 modes, else
// the line (any record format; NIN is the input-mode count, or the most there
// can be, then a.dec.nmodes - 1 of them are read).
template <int NIN, bool DEC>
__device__ __forceinline__ DecRec<NIN> any_rec(const MttkrpArgs& a, uint32_t i) {
  if constexpr (DEC) {
    return load_dec<NIN>(a.line, a.extra, i);
  } else {
    uint64_t lo, hi;
    DecRec<NIN> r;
    rec_read(a.line, a.dec.hi_words, i, lo, hi, r.v);
#pragma unroll
    for (int j = 0; j < NIN; ++j) {
      const int m = j < a.target ? j : j + 1;
      r.in[j] = m < a.dec.nmodes ? (uint32_t)line_field(lo, hi, a.dec.pos[m], a.dec.mask[m]) : 0;
    }
    r.row = (uint32_t)line_field(lo, hi, a.dec.pos[a.target], a.dec.mask[a.target]);
    return r;
  }
}

template <typename FT, int VW, int NIN, bool DEC, bool STAGE>
__global__ void __launch_bounds__(kMttkrpThreads, 4) any_walk_kernel(const MttkrpArgs a, int rank) {
  constexpr int V = 4, Q = V / VW;
  constexpr int U = NIN <= 3 ? 2 : 1;
  const int c0 = blockIdx.y * 32 * V;  // this window's first column
  const int cols = min(rank - c0, 32 * V);
  const int G = (cols + V - 1) / V, NPW = 32 / G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / G, sub = lane % G;
  const bool idle = grp >= NPW;
  // this lane's pieces: columns (q G + sub) VW of the window (a piece past
  // the last column reads the last one and is not written)
  int col[Q];
  bool mine[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int c = (q * G + sub) * VW;
    mine[q] = c < cols && !idle;
    col[q] = c0 + min(c, cols - VW);
  }
  extern __shared__ float any_smem[];  // STAGE: the output's rows, this window's columns
  if constexpr (STAGE) {
    for (int p = threadIdx.x; p < a.stage_rows * cols; p += kMttkrpThreads) any_smem[p] = 0.f;
    __syncthreads();
  }
  const uint32_t last = a.nnz - 1;
  const uint32_t ct = a.chunk_tiles ? a.chunk_tiles : 1;
  const uint32_t nchunks = (a.ntiles + ct - 1) / ct;
  const char* base[NIN];
#pragma unroll
  for (int j = 0; j < NIN; ++j) base[j] = static_cast<const char*>(a.in.f[j]);
  const size_t row_bytes = (size_t)rank * sizeof(FT);
  for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
    uint32_t cur = kNoRow;
    float acc[V];
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = 0.f;
    auto flush = [&]() {
      if constexpr (STAGE) {
        float* o = any_smem + (size_t)cur * cols - c0;
#pragma unroll
        for (int q = 0; q < V; ++q)
          if (mine[q / VW]) atomicAdd(o + col[q / VW] + q % VW, acc[q]);
      } else {
        float* o = a.out + (size_t)cur * rank;
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if (mine[q]) any_flush<VW>(o + col[q], acc + q * VW);
      }
    };
    const uint32_t t_end = min(c * ct + ct, a.ntiles);
    for (uint32_t tile = c * ct; tile < t_end; ++tile) {
      const uint32_t ts = tile * a.tile_nnz;
      const uint32_t te = min(ts + a.tile_nnz, a.nnz);
      const uint32_t chunk = (te - ts + kMttkrpWarps - 1) / kMttkrpWarps;
      const uint32_t ws = min(ts + warp * chunk, te);
      const uint32_t we = min(ws + chunk, te);
      const uint32_t sublen = (we - ws + NPW - 1) / NPW;
      const uint32_t gs = min(ws + grp * sublen, we);
      const uint32_t ge = idle ? gs : min(gs + sublen, we);
      DecRec<NIN> rec[U];
#pragma unroll
      for (int u = 0; u < U; ++u) rec[u] = any_rec<NIN, DEC>(a, min(gs + u, last));
      for (uint32_t i = gs, k = 0; k < sublen; k += U, i += U) {
        float f[U][NIN][V];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < NIN; ++j) {
            if (NIN > 4 && j + 1 >= a.dec.nmodes) continue;
            const char* p = base[j] + rec[u].in[j] * row_bytes;
#pragma unroll
            for (int q = 0; q < Q; ++q) any_piece<FT, VW>(p + col[q] * sizeof(FT), &f[u][j][q * VW]);
          }
        uint32_t rows[U];
        float vals[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          rows[u] = rec[u].row;
          vals[u] = rec[u].v;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) rec[u] = any_rec<NIN, DEC>(a, min(i + U + u, last));
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (i + u >= ge) continue;
          if (rows[u] != cur) {
            if (cur != kNoRow) flush();
            cur = rows[u];
#pragma unroll
            for (int q = 0; q < V; ++q) acc[q] = 0.f;
          }
#pragma unroll
          for (int q = 0; q < V; ++q) {
            float x = vals[u];
#pragma unroll
            for (int j = 0; j < NIN; ++j)
              if (NIN <= 4 || j + 1 < a.dec.nmodes) x *= f[u][j][q];
            acc[q] += x;
          }
        }
      }
    }
    const bool one = NPW > 1 && merge_groups<V>(cur, acc, G, NPW, lane);
    if (cur != kNoRow && !(one && grp)) flush();
  }
  if constexpr (STAGE) {
    __syncthreads();
    for (int p = threadIdx.x; p < a.stage_rows * cols; p += kMttkrpThreads)
      if (any_smem[p] != 0.f) atomicAdd(a.out + (size_t)(p / cols) * rank + c0 + p % cols, any_smem[p]);
  }
}

static int g_num_sms = 0;

static int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

static uint64_t l2_bytes() {
  static int bytes = 0;
  if (!bytes) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&bytes, cudaDevAttrL2CacheSize, dev);
    if (bytes <= 0) bytes = 126 << 20;
  }
  return (uint64_t)bytes;
}

// Tiles per chunk of the direct walks: up to kChunkTilesMax, keeping at
// least kChunksPerBlock chunks per block so the round robin still balances
// the blocks.
constexpr uint32_t kChunkTilesMax = 8;
constexpr uint32_t kChunksPerBlock = 8;
static uint32_t chunk_tiles_for(uint32_t ntiles, unsigned grid) {
  uint32_t c = kChunkTilesMax;
  while (c > 1 && (uint64_t)ntiles < (uint64_t)c * grid * kChunksPerBlock) c >>= 1;
  return c;
}

// The tiles of a walk that has no use for their intervals: sized so that
// `grid` blocks get the same number of equal tiles (the tensor's own tiles leave
// a last wave that is nearly empty: 489 tiles of 2048 on 444 blocks at 1M
// nonzeros), at most `most` nonzeros each, in multiples of `unit` (one step
// of every lane group of a block).
constexpr uint32_t kWalkTile = 4096;
constexpr uint32_t kDetTile = 16384;  // (a deterministic tile ends in a barrier)
constexpr unsigned kDetSms = 144;     // (a constant: the cut must not depend on the device; a few SMs left
                                      // for what runs beside the walk in a stream group)
static uint64_t tile_rounds(const MttkrpArgs& a, unsigned grid, uint32_t most) {  // tiles of a block
  const uint64_t wave = (uint64_t)grid * most;
  return std::max<uint64_t>(((uint64_t)a.nnz + wave - 1) / wave, 1);
}
static void cut_tiles(MttkrpArgs* a, unsigned grid, uint32_t unit, uint64_t rounds) {
  const uint64_t per = (a->nnz + grid * rounds - 1) / (grid * rounds);
  a->tile_nnz = (uint32_t)std::max<uint64_t>((per + unit - 1) / unit * unit, unit);
  a->ntiles = (uint32_t)(((uint64_t)a->nnz + a->tile_nnz - 1) / a->tile_nnz);
}
static void even_tiles(MttkrpArgs* a, unsigned grid, uint32_t unit, uint32_t most = kWalkTile) {
  cut_tiles(a, grid, unit, tile_rounds(*a, grid, most));
}
// The same with the blocks' tiles in equal chunks of up to kChunkTilesMax, at
// least `chunks` of them a block; returns the tiles of a chunk.  A hot row is
// updated once per warp and chunk, so short chunks lengthen the chain of its
// atomics, long ones the chains in registers.  Five of the walk with five blocks
// an SM are as long as eight of the walk with three, whose error they keep; two
// measured up to a sixth faster (4 modes, rank 16, 40M nonzeros: 495 us against
// 584) with up to a fifth more error (1000 rows of 20,000: 2.7e-7 against 2.4e-7).
static uint32_t even_chunks(MttkrpArgs* a, unsigned grid, uint32_t unit, uint32_t chunks) {
  uint64_t rounds = tile_rounds(*a, grid, kWalkTile);
  uint32_t c = kChunkTilesMax;
  while (c > 1 && rounds < (uint64_t)c * chunks) c >>= 1;
  rounds = (rounds + c - 1) / c * c;
  cut_tiles(a, grid, unit, rounds);
  return c;
}

template <int R, typename FT, int HW, bool STAGE, int NM>
static alto_status launch_tile(const MttkrpArgs& a, cudaStream_t st) {
  MttkrpArgs b = a;
  b.stage_rows = STAGE ? kStageBytes / (R * 4) : 0;
  const size_t smem = STAGE ? (size_t)kStageBytes : 0;
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    if (STAGE)
      ALTO_TRY_CUDA(cudaFuncSetAttribute(mttkrp_tile_kernel<R, FT, HW, STAGE, NM, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kStageBytes));
    else  // no shared memory: all of the unified L1 / shared storage as L1 (factor rows hit it)
      ALTO_TRY_CUDA(cudaFuncSetAttribute(mttkrp_tile_kernel<R, FT, HW, STAGE, NM, false>,
                                         cudaFuncAttributePreferredSharedMemoryCarveout, 0));
    ALTO_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &blocks_per_sm, mttkrp_tile_kernel<R, FT, HW, STAGE, NM, false>, kMttkrpThreads, smem));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  unsigned grid = std::min<unsigned>(a.ntiles, (unsigned)(num_sms() * blocks_per_sm));
  if (!grid) return ALTO_OK;
  b.chunk_tiles = chunk_tiles_for(a.ntiles, grid);
  mttkrp_tile_kernel<R, FT, HW, STAGE, NM, false><<<grid, kMttkrpThreads, smem, st>>>(b);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

template <int R, typename FT, int HW, int NM>
static alto_status launch_tma(const MttkrpArgs& a, int* err, cudaStream_t st) {
  const size_t smem = 2 * (size_t)kLineTile * (HW == 2 ? 32 : 16);
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    ALTO_TRY_CUDA(cudaFuncSetAttribute(mttkrp_tma_kernel<R, FT, HW, NM>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ALTO_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &blocks_per_sm, mttkrp_tma_kernel<R, FT, HW, NM>, kMttkrpThreads, smem));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  const unsigned ntiles = (a.nnz + kLineTile - 1) / kLineTile;
  const unsigned grid = std::min<unsigned>(ntiles, (unsigned)(num_sms() * blocks_per_sm));
  if (!grid) return ALTO_OK;
  mttkrp_tma_kernel<R, FT, HW, NM><<<grid, kMttkrpThreads, smem, st>>>(a, err);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

template <int R, typename FT, int NIN, bool DEEP = false>
static alto_status launch_walk(const MttkrpArgs& a, cudaStream_t st) {
  if constexpr (kCanBeDeep<R, FT, NIN> && !DEEP)
    if (a.nnz >= kDeepNnz && a.in_rows * (R * sizeof(FT)) > l2_bytes()) return launch_walk<R, FT, NIN, true>(a, st);
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    // no shared memory: all of the unified L1 / shared storage as L1 (factor rows hit it)
    ALTO_TRY_CUDA(cudaFuncSetAttribute(walk_kernel<R, FT, NIN, DEEP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       0));
    ALTO_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, walk_kernel<R, FT, NIN, DEEP>,
                                                                kMttkrpThreads, 0));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  if (!a.nnz) return ALTO_OK;
  MttkrpArgs b = a;
  using C = WalkCfg<R, FT, NIN, false, DEEP>;
  const unsigned full = (unsigned)(num_sms() * blocks_per_sm);
  b.chunk_tiles = even_chunks(&b, full, kMttkrpWarps * WalkMap<R, FT, C::V>::NPW * C::U, DEEP ? kChunksPerBlock : 5);
  const unsigned grid = std::min<unsigned>(b.ntiles, full);
  walk_kernel<R, FT, NIN, DEEP><<<grid, kMttkrpThreads, 0, st>>>(b);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// A line's output mode of few rows is summed in shared memory, block by block, where
// the rank is no multiple of four: a lane group's update is then two to four
// atomics, and these lengthen the chain of a hot row (6 modes, 500,000 nonzeros, 70
// rows: rank 3 391 us, a warp per nonzero 273, so 23; rank 10 165, 136 and 37).
// Fewer blocks where each would update the rows more often than it has nonzeros for
// them, as long as its groups have at most two steps (20,000 nonzeros, 70 rows,
// rank 3: 24.8 us, a warp per nonzero 14.9, so 9.3; with up to four steps 300 rows at
// rank 10 took 11.4 us instead of 8.4).
constexpr uint64_t kAnyStageBytes = 32 << 10;
constexpr uint64_t kAnyStageSteps = 2;

template <typename FT, int VW, int NIN, bool DEC>
static alto_status launch_any(const MttkrpArgs& a, int rank, cudaStream_t st) {
  const unsigned windows = (unsigned)((rank + 127) / 128);
  if (!a.nnz) return ALTO_OK;
  MttkrpArgs b = a;
  unsigned full = (unsigned)num_sms() * 4;
  const uint64_t cols = std::min(rank, 128), groups = kMttkrpWarps * (32 / ((cols + 3) / 4));
  b.stage_rows = 0;
  if (!DEC && VW < 4 && a.out_rows * cols * 4 <= kAnyStageBytes) {
    const uint64_t few = std::min<uint64_t>(std::max<uint64_t>(a.nnz / a.out_rows, 1), full);
    if (few == full || a.nnz <= kAnyStageSteps * groups * few) {
      full = (unsigned)few;
      b.stage_rows = (int)a.out_rows;
    }
  }
  even_tiles(&b, full, kMttkrpWarps);  // (the unit is a nonzero a warp: short walks want the blocks)
  const unsigned grid = std::min<unsigned>(b.ntiles, full);
  b.chunk_tiles = chunk_tiles_for(b.ntiles, grid);
  const dim3 blocks(grid, windows);
  if constexpr (!DEC && VW < 4) {
    if (b.stage_rows) {
      any_walk_kernel<FT, VW, NIN, false, true><<<blocks, kMttkrpThreads, b.stage_rows * cols * 4, st>>>(b, rank);
      ALTO_LAUNCHED();
      return ALTO_OK;
    }
  }
  any_walk_kernel<FT, VW, NIN, DEC, false><<<blocks, kMttkrpThreads, 0, st>>>(b, rank);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

template <typename FT, int VW>
static alto_status launch_any_modes(const MttkrpArgs& a, int rank, bool decoded, cudaStream_t st) {
  switch (a.dec.nmodes) {
    case 3: return decoded ? launch_any<FT, VW, 2, true>(a, rank, st) : launch_any<FT, VW, 2, false>(a, rank, st);
    case 4: return decoded ? launch_any<FT, VW, 3, true>(a, rank, st) : launch_any<FT, VW, 3, false>(a, rank, st);
    case 5: return decoded ? launch_any<FT, VW, 4, true>(a, rank, st) : launch_any<FT, VW, 4, false>(a, rank, st);
    default: return launch_any<FT, VW, ALTO_MAX_MODES - 1, false>(a, rank, st);
  }
}

// The widest load (4, 2 or 1 factors) that divides the rank and that the
// factors and the output are aligned for.
template <typename FT>
static alto_status launch_any_width(const MttkrpArgs& a, int rank, bool decoded, cudaStream_t st) {
  uintptr_t bits = reinterpret_cast<uintptr_t>(a.out) | ((uintptr_t)rank * 4);
  for (int j = 0; j + 1 < a.dec.nmodes; ++j)
    bits |= (reinterpret_cast<uintptr_t>(a.in.f[j]) | ((uintptr_t)rank * sizeof(FT))) * (4 / sizeof(FT));
  if (bits % 16 == 0) return launch_any_modes<FT, 4>(a, rank, decoded, st);
  if (bits % 8 == 0) return launch_any_modes<FT, 2>(a, rank, decoded, st);
  return launch_any_modes<FT, 1>(a, rank, decoded, st);
}

// The fix-up kernels of a deterministic MTTKRP whose walk left nslots slots.
static alto_status launch_det_fix(const MttkrpArgs& a, uint32_t nslots, int R, const DetLong& dl, cudaStream_t st) {
  const unsigned g1 = std::min<unsigned>((nslots + 7) / 8, (unsigned)num_sms() * 16);
  det_fix_short_kernel<<<g1, 256, 0, st>>>(a.det_rows, a.det_vals, nslots, R, a.out, dl);
  ALTO_LAUNCHED();
  det_fix_seg_kernel<<<(unsigned)num_sms() * 4, 256, 0, st>>>(a.det_vals, R, dl);
  ALTO_LAUNCHED();
  det_fix_final_kernel<<<(unsigned)num_sms(), 256, 0, st>>>(a.det_rows, R, a.out, dl);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// Deterministic MTTKRP (float32 factors, the specialised ranks): the walk of
// the row-sorted copy, then the fix-up of its chunks' slots.
template <int R, int NIN>
static alto_status launch_det_walk(const DetItem& it, cudaStream_t st) {
  if (!it.nblocks) return ALTO_OK;
  det_walk_kernel<R, NIN><<<it.nblocks, kMttkrpThreads, 0, st>>>(it.a);
  ALTO_LAUNCHED();
  det_fix_kernel<<<std::min<unsigned>(it.nslots, (unsigned)num_sms() * 8), 256, 0, st>>>(it.a, it.nslots, R);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

// As launch_det_walk on lines that are not decoded (2 modes, or more than 5).
template <int R, int HW>
static alto_status launch_det_line(const DetItem& it, cudaStream_t st) {
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    ALTO_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &blocks_per_sm, mttkrp_tile_kernel<R, float, HW, false, ALTO_MAX_MODES, true>, kMttkrpThreads, 0));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  const unsigned grid = std::min<unsigned>(it.a.ntiles, (unsigned)(num_sms() * blocks_per_sm));
  if (!grid) return ALTO_OK;
  mttkrp_tile_kernel<R, float, HW, false, ALTO_MAX_MODES, true><<<grid, kMttkrpThreads, 0, st>>>(it.a);
  ALTO_LAUNCHED();
  return launch_det_fix(it.a, it.nslots, R, it.dl, st);
}

template <int R>
static alto_status launch_det(const DetItem& it, cudaStream_t st) {
  if (it.hw == kDecoded) {
    switch (it.a.dec.nmodes) {
      case 3: return launch_det_walk<R, 2>(it, st);
      case 4: return launch_det_walk<R, 3>(it, st);
      default: return launch_det_walk<R, 4>(it, st);
    }
  }
  if (it.hw == 0) return launch_det_line<R, 0>(it, st);
  if (it.hw == 1) return launch_det_line<R, 1>(it, st);
  return launch_det_line<R, 2>(it, st);
}

static alto_status launch_det_rank(const DetItem& it, int rank, cudaStream_t st) {
  switch (rank) {
    case 8: return launch_det<8>(it, st);
    case 16: return launch_det<16>(it, st);
    case 32: return launch_det<32>(it, st);
    case 64: return launch_det<64>(it, st);
    case 128: return launch_det<128>(it, st);
    default: break;
  }
  set_error("the deterministic MTTKRP takes rank 8, 16, 32, 64 or 128 (got %d)", rank);
  return ALTO_ERR_UNSUPPORTED;
}

template <int R, int NIN>
static uint32_t det_unit_nm() {
  using C = WalkCfg<R, float, NIN, true>;
  return kMttkrpWarps * WalkMap<R, float, C::V>::NPW * C::U;
}
// Nonzeros of one step of every lane group of a deterministic walk's block.
template <int R>
static uint32_t det_unit(int nmodes) {
  return nmodes == 3 ? det_unit_nm<R, 2>() : nmodes == 4 ? det_unit_nm<R, 3>() : det_unit_nm<R, 4>();
}
static uint32_t det_unit_of(int rank, int nmodes) {
  switch (rank) {
    case 8: return det_unit<8>(nmodes);
    case 16: return det_unit<16>(nmodes);
    case 32: return det_unit<32>(nmodes);
    case 64: return det_unit<64>(nmodes);
    default: return det_unit<128>(nmodes);
  }
}

// Lane groups per warp of the deterministic walk of a line that is not decoded.
static uint32_t groups_per_warp(int rank) {
  switch (rank) {
    case 8: return LaneWidth<8>::NPW;
    case 16: return LaneWidth<16>::NPW;
    case 32: return LaneWidth<32>::NPW;
    case 64: return LaneWidth<64>::NPW;
    default: return LaneWidth<128>::NPW;
  }
}

bool deterministic_supported(int rank, alto_dtype fdtype) {
  return fdtype == ALTO_F32 && (rank == 8 || rank == 16 || rank == 32 || rank == 64 || rank == 128);
}

// The ALTO line (or a copy that keeps its record format).
template <int R, typename FT, int HW>
static alto_status launch_modes(const MttkrpArgs& a, bool stage, bool bulk_feed, int* err, cudaStream_t st) {
#define NM_CASE(NN)                                                                   \
  case NN:                                                                            \
    if (stage) return launch_tile<R, FT, HW, true, NN>(a, st);                        \
    return bulk_feed ? launch_tma<R, FT, HW, NN>(a, err, st) : launch_tile<R, FT, HW, false, NN>(a, st);
  switch (a.dec.nmodes) {
    NM_CASE(3)
    NM_CASE(4)
    NM_CASE(5)
    default:
      return stage ? launch_tile<R, FT, HW, true, ALTO_MAX_MODES>(a, st)
                   : launch_tile<R, FT, HW, false, ALTO_MAX_MODES>(a, st);
  }
#undef NM_CASE
}

// hw: the record format of the line walked.  The specialised ranks need
// 16-byte aligned rows (8 for bfloat16); any other call takes the any-rank walk.
template <int R, typename FT>
static alto_status launch_specialised(const MttkrpArgs& a, int hw, bool stage, bool bulk_feed, int* err,
                                      cudaStream_t st) {
  if (hw == kDecoded) {
    switch (a.dec.nmodes) {
      case 3: return launch_walk<R, FT, 2>(a, st);
      case 4: return launch_walk<R, FT, 3>(a, st);
      default: return launch_walk<R, FT, 4>(a, st);
    }
  }
  if (hw == 0) return launch_modes<R, FT, 0>(a, stage, bulk_feed, err, st);
  if (hw == 1) return launch_modes<R, FT, 1>(a, stage, bulk_feed, err, st);
  return launch_modes<R, FT, 2>(a, stage, bulk_feed, err, st);
}

template <typename FT>
static alto_status launch_rank(const MttkrpArgs& a, int rank, int hw, bool stage, bool bulk_feed, uintptr_t misalign,
                               int* err, cudaStream_t st) {
  // (the decoded walk reads bfloat16 rows in 16-byte pieces)
  const bool aligned = misalign % 16 == 0 || (sizeof(FT) == 2 && hw != kDecoded && misalign % 8 == 0);
  if (aligned) {
    switch (rank) {
      case 8: return launch_specialised<8, FT>(a, hw, stage, bulk_feed, err, st);
      case 16: return launch_specialised<16, FT>(a, hw, stage, bulk_feed, err, st);
      case 32: return launch_specialised<32, FT>(a, hw, stage, bulk_feed, err, st);
      case 64: return launch_specialised<64, FT>(a, hw, stage, bulk_feed, err, st);
      case 128: return launch_specialised<128, FT>(a, hw, stage, bulk_feed, err, st);
      default: break;
    }
  }
  return launch_any_width<FT>(a, rank, hw == kDecoded, st);
}

// Fraction of the mode's tiles whose output interval fits the staging buffer
// at this rank and is at most half the tile (so staging saves updates).
static double stageable_fraction(const alto_tensor* t, int mode, int rank) {
  const auto& v = t->tile_len_sorted[mode];
  if (v.empty()) return 0.0;
  const uint32_t cap = std::min<uint32_t>(kStageBytes / (rank * 4), t->tile_nnz / 2);
  const size_t n = std::upper_bound(v.begin(), v.end(), cap) - v.begin();
  return (double)n / (double)v.size();
}

static const TuneEntry* tuned_entry(const alto_tensor* t, int mode, int rank, alto_dtype fdtype) {
  for (const auto& e : t->tuned)
    if (e.mode == mode && e.rank == rank && e.fdtype == (int)fdtype) return &e;
  return nullptr;
}

bool mttkrp_tuned(const alto_tensor* t, int mode, int rank, alto_dtype fdtype) {
  return tuned_entry(t, mode, rank, fdtype) != nullptr;
}

alto_mttkrp_variant unsorted_variant(const alto_tensor* t, int mode, int rank) {
  if (mode == t->stream_mode && t->dims[mode] * rank * 4 <= (uint64_t)kStageBytes) return ALTO_MTTKRP_STREAM;
  if (stageable_fraction(t, mode, rank) >= 0.5) return ALTO_MTTKRP_STAGED;
  return ALTO_MTTKRP_ATOMIC;
}

alto_mttkrp_variant choose_variant(const alto_tensor* t, int mode, int rank, alto_dtype fdtype) {
  if (const TuneEntry* e = tuned_entry(t, mode, rank, fdtype)) return e->variant;
  // The reference's rule (include/alto.hpp:835-846) picks atomics for long
  // low-reuse modes, the stream kernel for the stream mode and da_mem
  // otherwise.  On the device: stage where the tiles' intervals fit, walk a
  // row-sorted copy where rows are reused but the intervals are too wide,
  // else plain vector atomics.
  const alto_mttkrp_variant v = unsorted_variant(t, mode, rank);
  const uint64_t reuse = t->dims[mode] ? t->nnz / t->dims[mode] : 0;
  return v == ALTO_MTTKRP_ATOMIC && reuse > 4 ? ALTO_MTTKRP_SORTED : v;
}

// The arguments of a walk of mode `mode` into `out`: of the line, or of the
// mode's row-sorted copy (built if it is not there); *hw its record format.
static alto_status fill_args(alto_tensor* t, int mode, const void* const* factors, float* out, bool sorted,
                             MttkrpArgs* args, int* hw, cudaStream_t st) {
  MttkrpArgs& a = *args;
  a.line = t->line.p;
  a.extra = nullptr;
  a.tile_iv = t->tile_iv.as<uint32_t>();
  a.ntiles = t->nnz ? t->ntiles : 0;
  *hw = t->dec.hi_words;
  if (sorted && t->nnz) {
    if (!t->sorted[mode].ready || t->sorted[mode].for_nnz != t->nnz) ALTO_TRY(build_sorted_line(t, mode, st));
    const SortedLine& s = t->sorted[mode];
    a.line = s.line.p;
    a.extra = s.extra.p;
    a.tile_iv = s.tile_iv.as<uint32_t>();
    a.ntiles = s.ntiles;
    *hw = s.hw;
  }
  a.nnz = (uint32_t)t->nnz;
  a.tile_nnz = t->tile_nnz;
  a.target = mode;
  a.dec = t->dec;
  a.out = out;
  int j = 0;
  a.in_rows = 0;
  a.out_rows = t->dims[mode];
  for (int m = 0; m < t->nmodes; ++m) {
    a.fac.f[m] = factors[m];
    if (m == mode) continue;
    a.in.f[j++] = factors[m];
    a.in_rows += t->dims[m];
  }
  return ALTO_OK;
}

alto_status run_mttkrp(alto_tensor* t, int mode, const void* const* factors, alto_dtype fdtype,
                       int rank, float* out, int accumulate, alto_mttkrp_variant variant,
                       cudaStream_t st) {
  return run_mttkrp_feed(t, mode, factors, fdtype, rank, out, accumulate, variant, -1, st);
}

// feed: 1 streams the line through shared memory by bulk copy (a line that is
// not decoded), 0 loads it directly, -1 uses the autotuned choice (direct
// when untuned).
alto_status run_mttkrp_feed(alto_tensor* t, int mode, const void* const* factors, alto_dtype fdtype,
                            int rank, float* out, int accumulate, alto_mttkrp_variant variant, int feed,
                            cudaStream_t st) {
  if (feed < 0) {
    const TuneEntry* e = variant == ALTO_MTTKRP_AUTO ? tuned_entry(t, mode, rank, fdtype) : nullptr;
    feed = e ? e->feed : 0;
  }
  if (variant == ALTO_MTTKRP_AUTO) variant = choose_variant(t, mode, rank, fdtype);
  const bool det = variant == ALTO_MTTKRP_DETERMINISTIC;
  if (det && !deterministic_supported(rank, fdtype)) {
    set_error("the deterministic MTTKRP takes float32 factors at rank 8, 16, 32, 64 or 128");
    return ALTO_ERR_UNSUPPORTED;
  }
  if (!accumulate)
    ALTO_TRY_CUDA(cudaMemsetAsync(out, 0, (size_t)t->dims[mode] * rank * sizeof(float), st));
  if (!t->nnz) return ALTO_OK;
  if (det) {
    DetItem it;
    ALTO_TRY(det_prepare(t, mode, factors, rank, out, &it, st));
    it.a.det_add = accumulate ? 1 : 0;
    return launch_det_rank(it, rank, st);
  }
  MttkrpArgs a{};
  int hw = t->dec.hi_words;  // record format of the line walked
  ALTO_TRY(fill_args(t, mode, factors, out, variant == ALTO_MTTKRP_SORTED, &a, &hw, st));
  // the low address bits of the output and the input factors
  uintptr_t misalign = reinterpret_cast<uintptr_t>(out);
  uintptr_t fac_bits = 0;
  for (int m = 0; m < t->nmodes; ++m)
    if (m != mode) fac_bits |= reinterpret_cast<uintptr_t>(factors[m]);
  const bool stage = variant == ALTO_MTTKRP_STAGED || variant == ALTO_MTTKRP_STREAM;
  ALTO_TRY(ensure_error_words(t, st));
  int* err = t->err.as<int>();
  const bool bulk = feed == 1;
  if (fdtype == ALTO_BF16) {
    if (misalign % 16) fac_bits |= 1;  // (float4 updates of the output)
    return launch_rank<__nv_bfloat16>(a, rank, hw, stage, bulk, fac_bits % 16, err, st);
  }
  return launch_rank<float>(a, rank, hw, stage, bulk, (misalign | fac_bits) % 16, err, st);
}

alto_status det_prepare(alto_tensor* t, int mode, const void* const* factors, int rank, float* out, DetItem* item,
                        cudaStream_t st) {
  if (!deterministic_supported(rank, ALTO_F32)) {
    set_error("the deterministic MTTKRP takes float32 factors at rank 8, 16, 32, 64 or 128");
    return ALTO_ERR_UNSUPPORTED;
  }
  MttkrpArgs a{};
  int hw = t->dec.hi_words;
  // (a mode of length 1 is already in row order in a line that is not decoded)
  ALTO_TRY(fill_args(t, mode, factors, out, t->dims[mode] > 1 || decoded_modes(t->nmodes), &a, &hw, st));
  bool aligned = (reinterpret_cast<uintptr_t>(out) % 16) == 0;
  for (int m = 0; m < t->nmodes; ++m)
    if (m != mode && (reinterpret_cast<uintptr_t>(factors[m]) % 16) != 0) aligned = false;
  if (!aligned) {
    set_error("the deterministic MTTKRP needs 16-byte aligned factors and output");
    return ALTO_ERR_UNSUPPORTED;
  }
  uint64_t nslots = (uint64_t)a.ntiles * kMttkrpWarps * groups_per_warp(rank) * 2;
  item->nblocks = 0;
  if (hw == kDecoded) {
    // a chunk per block, cut by nnz and rank alone (the order of the sums is a
    // function of them); small tiles for a small tensor, whose groups' chains of
    // dependent loads are what it waits for
    even_tiles(&a, 3 * kDetSms, det_unit_of(rank, t->nmodes), kDetTile);
    a.chunk_tiles = (a.ntiles + 3 * kDetSms - 1) / (3 * kDetSms);
    if (!a.chunk_tiles) a.chunk_tiles = 1;
    item->nblocks = (a.ntiles + a.chunk_tiles - 1) / a.chunk_tiles;
    nslots = 2 * (uint64_t)item->nblocks;
  }
  ALTO_TRY(tensor_ensure(t, t->det_rows, std::max<uint64_t>(nslots, 1) * 4));
  ALTO_TRY(tensor_ensure(t, t->det_vals, std::max<uint64_t>(nslots, 1) * rank * 4));
  a.det_rows = t->det_rows.as<uint32_t>();
  a.det_vals = t->det_vals.as<float>();
  item->a = a;
  item->dl = DetLong{};
  if (hw != kDecoded) {
    // long chains: each has more than kShortChain slots; segments:
    // sum over chains of ceil(len / kChainSeg)
    const uint64_t max_chains = nslots / (kShortChain + 1) + 1;
    const uint64_t max_segs = nslots / kChainSeg + max_chains;
    auto up = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
    const uint64_t o_chains = 256, o_segs = o_chains + up(max_chains * sizeof(uint4)),
                   o_part = o_segs + up(max_segs * sizeof(uint2)), bytes = o_part + max_segs * rank * 4;
    const size_t before = t->det_long.bytes;  // a new allocation starts with zero counters
    ALTO_TRY(tensor_ensure(t, t->det_long, bytes));
    if (t->det_long.bytes != before) ALTO_TRY_CUDA(cudaMemsetAsync(t->det_long.p, 0, 16, st));
    char* base = t->det_long.as<char>();
    item->dl = DetLong{reinterpret_cast<uint32_t*>(base), reinterpret_cast<uint4*>(base + o_chains),
                       reinterpret_cast<uint2*>(base + o_segs), reinterpret_cast<float*>(base + o_part)};
  }
  item->nslots = (uint32_t)nslots;
  item->hw = hw;
  item->out_floats = t->dims[mode] * (uint64_t)rank;
  item->active = nullptr;
  return ALTO_OK;
}

template <int R, int NIN>
static alto_status det_group_nm(Strided<DetItem> items, const uint32_t* tile_off, cudaStream_t st) {
  static int blocks_per_sm = 0;
  if (!blocks_per_sm) {
    ALTO_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, det_tile_group_kernel<R, NIN>,
                                                                kMttkrpThreads, 0));
    if (blocks_per_sm < 1) blocks_per_sm = 1;
  }
  const unsigned sm = (unsigned)num_sms();
  det_tile_group_kernel<R, NIN><<<sm * blocks_per_sm, kMttkrpThreads, 0, st>>>(items, tile_off);
  ALTO_LAUNCHED();
  det_fix_group_kernel<<<sm * 8, 256, 0, st>>>(items, R);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

alto_status det_group_zero(Strided<DetItem> items, cudaStream_t st) {
  det_zero_group_kernel<<<(unsigned)num_sms() * 4, 256, 0, st>>>(items);
  ALTO_LAUNCHED();
  return ALTO_OK;
}

template <int R>
static alto_status det_group_rank(Strided<DetItem> items, const uint32_t* tile_off, int hw, int nmodes,
                                  cudaStream_t st) {
  if (hw == kDecoded && nmodes == 3) return det_group_nm<R, 2>(items, tile_off, st);
  if (hw == kDecoded && nmodes == 4) return det_group_nm<R, 3>(items, tile_off, st);
  if (hw == kDecoded && nmodes == 5) return det_group_nm<R, 4>(items, tile_off, st);
  set_error("grouped MTTKRP: record format %d with %d modes is not supported", hw, nmodes);
  return ALTO_ERR_UNSUPPORTED;
}

alto_status det_group_launch(Strided<DetItem> items, const uint32_t* tile_off, int rank, int hw, int nmodes,
                             cudaStream_t st) {
  switch (rank) {
    case 8: return det_group_rank<8>(items, tile_off, hw, nmodes, st);
    case 16: return det_group_rank<16>(items, tile_off, hw, nmodes, st);
    case 32: return det_group_rank<32>(items, tile_off, hw, nmodes, st);
    case 64: return det_group_rank<64>(items, tile_off, hw, nmodes, st);
    default: break;
  }
  set_error("grouped MTTKRP: rank %d is not supported (8, 16, 32 or 64)", rank);
  return ALTO_ERR_UNSUPPORTED;
}

// One block: whether two records kLongRun apart, kLongRun * k and the next, have
// one row (nnz / kLongRun reads).
template <int NIN>
__global__ void __launch_bounds__(256)
    long_run_kernel(const void* __restrict__ line, const void* __restrict__ extra, uint64_t nnz, int* __restrict__ found) {
  int any = 0;
  for (uint64_t i = (uint64_t)threadIdx.x * kLongRun; i + kLongRun < nnz; i += 256ull * kLongRun)
    any |= load_dec<NIN>(line, extra, (uint32_t)i).row == load_dec<NIN>(line, extra, (uint32_t)(i + kLongRun)).row;
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) *found = any;
}

alto_status sorted_long_runs(alto_tensor* t, int mode, bool* found, cudaStream_t st) {
  SortedLine& s = t->sorted[mode];
  if (s.long_runs < 0) {
    DevBuf flag;
    ALTO_TRY(flag.ensure(sizeof(int)));
    const void *line = s.line.p, *extra = s.extra.p;
    if (t->nmodes == 3) long_run_kernel<2><<<1, 256, 0, st>>>(line, extra, t->nnz, flag.as<int>());
    if (t->nmodes == 4) long_run_kernel<3><<<1, 256, 0, st>>>(line, extra, t->nnz, flag.as<int>());
    if (t->nmodes == 5) long_run_kernel<4><<<1, 256, 0, st>>>(line, extra, t->nnz, flag.as<int>());
    ALTO_LAUNCHED();
    int any = 0;
    ALTO_TRY_CUDA(cudaMemcpyAsync(&any, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    ALTO_TRY_CUDA(cudaStreamSynchronize(st));
    s.long_runs = any;
  }
  *found = s.long_runs != 0;
  return ALTO_OK;
}

// Time every applicable variant once per mode (after one warm run) into a
// scratch output and record the fastest for ALTO_MTTKRP_AUTO.  Synchronous;
// not for use inside stream capture.
alto_status autotune(alto_tensor* t, const void* const* factors, alto_dtype fdtype, int rank,
                     cudaStream_t st, alto_mttkrp_variant* chosen) {
  uint64_t max_dim = 0;
  for (int m = 0; m < t->nmodes; ++m) max_dim = std::max<uint64_t>(max_dim, t->dims[m]);
  DevBuf out;
  ALTO_TRY(out.ensure(max_dim * rank * 4));
  cudaEvent_t e0, e1;
  ALTO_TRY_CUDA(cudaEventCreate(&e0));
  ALTO_TRY_CUDA(cudaEventCreate(&e1));
  std::vector<TuneEntry> keep;
  for (const auto& e : t->tuned)
    if (!(e.rank == rank && e.fdtype == (int)fdtype)) keep.push_back(e);
  t->tuned = keep;
  alto_status status = ALTO_OK;
  for (int m = 0; m < t->nmodes && status == ALTO_OK; ++m) {
    struct Cand {
      alto_mttkrp_variant v;
      int feed;
    };
    const Cand cands[] = {{ALTO_MTTKRP_ATOMIC, 0}, {ALTO_MTTKRP_ATOMIC, 1}, {ALTO_MTTKRP_STAGED, 0},
                          {ALTO_MTTKRP_SORTED, 0}};
    alto_mttkrp_variant best = ALTO_MTTKRP_ATOMIC;
    int best_feed = 0;
    float best_ms = 1e30f;
    for (const Cand& c : cands) {
      const alto_mttkrp_variant v = c.v;
      if (v == ALTO_MTTKRP_STAGED && stageable_fraction(t, m, rank) == 0.0) continue;
      if (v == ALTO_MTTKRP_SORTED && t->nnz / std::max<uint64_t>(t->dims[m], 1) < 2) continue;
      status = run_mttkrp_feed(t, m, factors, fdtype, rank, out.as<float>(), 0, v, c.feed, st);  // warm / build
      if (status != ALTO_OK) break;
      cudaEventRecord(e0, st);
      status = run_mttkrp_feed(t, m, factors, fdtype, rank, out.as<float>(), 0, v, c.feed, st);
      cudaEventRecord(e1, st);
      if (status != ALTO_OK) break;
      if (cudaEventSynchronize(e1) != cudaSuccess) {
        status = cuda_status(cudaGetLastError(), "autotune", __FILE__, __LINE__);
        break;
      }
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best_ms) {
        best_ms = ms;
        best = v;
        best_feed = c.feed;
      }
    }
    t->tuned.push_back({m, rank, (int)fdtype, best, best_feed});
    if (chosen) chosen[m] = best;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return status;
}

}  // namespace alto
