// knn_tc.cu -- the precision form of the fused kNN: tensor-core (tcgen05) distances in TF32,
// BF16, scaled FP16 or split BF16 (hi*hi + hi*lo + lo*hi), with FP32 accumulation in TMEM, followed by an
// FP64 re-rank of every candidate whose approximate distance lies within a rigorous rounding
// bound of the query's k-th approximate distance. The result is the exact FP64 top-k (ties to
// the lower id) of the caller's inputs, merged into the caller's heaps. Tables are float or double:
// double rows are centred in FP64 before they are rounded to the MMA format, and rows that leave
// the floats' range go back to the caller's CUDA-core path.
//
// Kernels (one call):
//   tc_center     partial sums of the shift vector mu = mean of a strided sample of candidate rows
//   tc_pack       candidates and queries: add the partial sums, gather, centre, round to the MMA
//                 format into a row-major [rows][d_pad] panel (TMA source), effective norm
//                 X2 - 2 mu.x + mu.mu (the centred norm, built on the caller's norm) in FP64,
//                 the terms of the error bound, ids; running maxima over the candidates
//   tc_knn        warp 0 TMA producer, warp 1 MMA issuer (TMEM owner), warps 2-9 epilogue (two
//                 per TMEM lane quarter, each taking half of every tile's columns) with one
//                 query row per thread: approximate d' = qn' + cn' - 2<q~,c~> (with the norm
//                 column, cn' enters through one extra MMA against an all-ones A tile and the
//                 accumulator holds w = -v/2); per row and epilogue part a sorted
//                 list of the ceil(k/2) smallest quad minima of its own columns in shared memory;
//                 any two such lists hold k candidates, so the second smallest root a row can see (its own, the
//                 other part's, and the roots up to three other splits published) bounds the
//                 k-th from above (threshold = that + 2E); per-query logs in HBM of every group of
//                 four adjacent candidates with one under the threshold
//   tc_rerank     one warp per query (tc_rerank_cta: one CTA per query, for few queries): exact
//                 FP64 distances of the logged band, sorted merge with the incoming heap row,
//                 descending write-back (a valid max-heap); tc_rerank_leaf (batching form) sorts
//                 and writes a row only if it changes
//   tc_fallback   queries whose log overflowed: exact FP64 brute force over all candidates
//
// Error bound (per query q, all candidates c; r(x) = |x - fmt(x)|, the norm of a row's rounding
// residual, measured per row; M = max |c~|, R = max r(c~), CN = max |cn'|, D = padded dimension,
// n = D + NORM_TERMS accumulated terms, u = unit roundoff of the MMA input format):
//   |d'(q,c) - d(q,c)| <= E_q = 1.25 * [ 2 (r(q~) M + (|q~| + r(q~)) R)          input rounding
//                                  + 2 (n 2^-23 (1+u)^2 + 2^-22) |q~| M          accumulation
//                                  + 3 * 2^-24 (CN + |qn'| + 2 |q~| M) ] + noise
// For the split format r(q~) M + ... is replaced by 3.2 u^2 |q~| M (u = 2^-8; it covers the omitted
// lo x lo product) and n = 3D + NORM_TERMS. With the norm column E gains 1.25 (t 2^-23 + 2^-24) CN
// for the norm parts it sums, t = NORM_TERMS in the split format, which accumulates them last, and n
// in the others. `noise` covers the rounding of the FP64 distance itself, (4d + 32) 2^-53 of
// the squared norms' scale. Measuring r takes the input term to about 0.4 of its worst case
// (2u + u^2) |q~| M.
#include "knn_common.cuh"
#include "knn_internal.h"
#include "tc_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace gsknn {
namespace tc {

constexpr int TC_M = 128;            // queries per CTA (TMEM lanes)
constexpr int CHIP_SMS = 148;        // B200: grids of the grid-stride kernels
constexpr int CHUNK_BYTES = 128;     // K bytes per TMA box / swizzle atom row
constexpr int A_CHUNK = TC_M * CHUNK_BYTES;  // 16 KB
// Warp 0 TMA producer, warp 1 MMA issuer, then NEPI epilogue warps: NPART per TMEM lane quarter,
// part j of a quarter taking the j-th of NPART equal column ranges of every tile. Every part keeps
// a small heap of its own columns per row (the partition bound, see TcParams::proot).
constexpr int NEPI = TC_EPI_WARPS;
constexpr int NPART = TC_EPI_PARTS;
constexpr int NTHREADS = 32 * (2 + NEPI);
constexpr uint32_t LOG_OVF = 1u << 30;
constexpr size_t LOG_ENTRY = sizeof(float4) + sizeof(uint32_t);  // a logged quad and its position
// The epilogue frees a TMEM accumulator as soon as its reads have landed, while it still uses
// the tile's candidate norms; the norms therefore get one slot more than the two accumulators
// (the slot the MMA warp refills belongs to a tile every epilogue warp has finished).
constexpr int CN_SLOTS = 3;

// ------------------------------------------------------------------------------------------
// shift vector
// ------------------------------------------------------------------------------------------
// The shift is the mean of a strided sample of the candidate rows, summed in a fixed order so that
// it is the same bits on every run: tc_center, on a grid of (dimension groups of 32, CENTER_SLICES
// slices of the sample), 16 warps per block, lane = dimension, warps striding over the slice's rows
// (coalesced row segments), writes one partial sum, minimum and maximum per (slice, dimension) and
// one row count per slice; tc_pack adds the partials in slice order, and takes the scale of the
// FP16 format from the widest dimension. Being the first kernel of a call it also clears
// the call's status word and the candidates' bound statistics.
constexpr int CENTER_SLICES = 16;
constexpr int CENTER_ROWS = 1024;  // sampled rows (any shift is valid; it only narrows the bound)
constexpr int CENTER_WARPS = 16;
constexpr int CENTER_PARTS = 3 * CENTER_SLICES;  // doubles per dimension

template <typename T>
__global__ void __launch_bounds__(32 * CENTER_WARPS) tc_center(
    const T *__restrict__ X, int d, long long nrows, const int *__restrict__ idx, int count,
    int nsample, double *__restrict__ part, int *__restrict__ part_n, unsigned *stats,
    int nstats, int *clear) {
  __shared__ double ps[CENTER_WARPS][33], pmn[CENTER_WARPS][33], pmx[CENTER_WARPS][33];
  __shared__ int pc[CENTER_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    if (stats && (int)threadIdx.x < nstats) stats[threadIdx.x] = 0u;
    if (clear && threadIdx.x == 0) *clear = 0;
  }
  const int p = blockIdx.x * 32 + lane;
  const int t_lo = (int)((long long)nsample * blockIdx.y / CENTER_SLICES);
  const int t_hi = (int)((long long)nsample * (blockIdx.y + 1) / CENTER_SLICES);
  double s = 0.0, mn = Num<double>::inf(), mx = -Num<double>::inf();
  int used = 0;
  // four sample rows per round: their index and row loads are independent and issue together
  for (int t0 = t_lo + warp; t0 < t_hi; t0 += CENTER_WARPS * 4) {
    T v[4];
    bool ok[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int t = t0 + CENTER_WARPS * u;
      long long row = -1;
      if (t < t_hi) row = idx[(long long)t * count / nsample];
      ok[u] = row >= 0 && row < nrows;
      v[u] = ok[u] && p < d ? X[row * d + p] : T(0);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (ok[u]) {
        if (p < d) {
          s += (double)v[u];
          mn = fmin(mn, (double)v[u]);
          mx = fmax(mx, (double)v[u]);
        }
        used++;
      }
    }
  }
  ps[warp][lane] = s;
  pmn[warp][lane] = mn;
  pmx[warp][lane] = mx;
  if (lane == 0) pc[warp] = used;
  __syncthreads();
  if (warp == 0) {
    double tot = 0.0;
    int n = 0;
    for (int w = 0; w < CENTER_WARPS; w++) {
      tot += ps[w][lane];
      mn = fmin(mn, pmn[w][lane]);
      mx = fmax(mx, pmx[w][lane]);
      n += pc[w];
    }
    if (p < d) {
      part[(size_t)blockIdx.y * d + p] = tot;
      part[(size_t)(CENTER_SLICES + blockIdx.y) * d + p] = mn;
      part[(size_t)(2 * CENTER_SLICES + blockIdx.y) * d + p] = mx;
    }
    if (blockIdx.x == 0 && lane == 0) part_n[blockIdx.y] = n;
  }
}

// ------------------------------------------------------------------------------------------
// packing
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// FP16 rounding with saturation; subnormals become 0 (the residual is measured either way).
__device__ __forceinline__ __half to_f16(float x) {
  const __half h = __float2half_rn(fminf(fmaxf(x, -65504.0f), 65504.0f));
  return fabsf(__half2float(h)) < 6.103515625e-5f ? __ushort_as_half(0) : h;
}

// Norm column of candidate row r (32 bytes, the K of one MMA): x = -cn/2 as the sum of three parts
// in the MMA input format, then zeros. Against an A tile whose rows all hold the parts' weights the
// MMA adds x to <q~, c~>, so the accumulator holds w = <q~, c~> - cn/2 = -v/2. A padding row holds
// -inf (w = -inf, v = +inf: never admitted). TF32 and BF16: weights 1, and the parts (3 x 11 and
// 3 x 8 significant bits) are exact for the 24 of the float. FP16: x in the panel's scale, weights
// 2^14, 2^3, 2^-8 for its narrow exponent; what the parts leave of x is returned.
__device__ __forceinline__ float write_norm_row(int fmt, void *npanel, int r, bool real, float x) {
  uint4 lo4 = make_uint4(0u, 0u, 0u, 0u), hi4 = make_uint4(0u, 0u, 0u, 0u);
  float rest = 0.0f;
  if (fmt == 0) {
    uint32_t h = 0xFF800000u, m = 0u, l = 0u;
    if (real) {
      h = to_tf32(x);
      const float r1 = x - __uint_as_float(h);
      m = to_tf32(r1);
      l = to_tf32(r1 - __uint_as_float(m));
    }
    lo4 = make_uint4(h, m, l, 0u);
  } else if (fmt == 3) {
    uint32_t h = 0xFC00u, m = 0u, l = 0u;
    if (real) {
      const __half a = to_f16(x * 6.103515625e-5f);
      const float r1 = x - __half2float(a) * 16384.0f;
      const __half b = to_f16(r1 * 0.125f);
      const float r2 = r1 - __half2float(b) * 8.0f;
      const __half c = to_f16(r2 * 256.0f);
      rest = fabsf(r2 - __half2float(c) * 0.00390625f);
      h = __half_as_ushort(a);
      m = __half_as_ushort(b);
      l = __half_as_ushort(c);
    }
    lo4 = make_uint4(h | (m << 16), l, 0u, 0u);
  } else {
    uint32_t h = 0xFF80u, m = 0u, l = 0u;
    if (real) {
      const __nv_bfloat16 bh = __float2bfloat16_rn(x);
      const float r1 = x - __bfloat162float(bh);
      const __nv_bfloat16 bm = __float2bfloat16_rn(r1);
      const __nv_bfloat16 bl = __float2bfloat16_rn(r1 - __bfloat162float(bm));
      h = __bfloat16_as_ushort(bh);
      m = __bfloat16_as_ushort(bm);
      l = __bfloat16_as_ushort(bl);
    }
    lo4 = make_uint4(h | (m << 16), l, 0u, 0u);
  }
  uint4 *dst = reinterpret_cast<uint4 *>(static_cast<char *>(npanel) + (size_t)r * 32);
  dst[0] = lo4;
  dst[1] = hi4;
  return rest;
}

// One side of a packing launch: `rows_pad` panel rows, of which the first `count` are points
// idx[r] (idx[rowmap[r]] with a row map) of table X. `dcount` (device) replaces `count` and limits
// the panel to the tiles it needs; `gate` (device) skips the side when it reads 0; `pad_ok` packs
// index -1 as an empty padding row instead of reporting it, and takes the point as its heap row.
template <typename T>
struct PackSide {
  const T *X, *X2;
  long long nrows;
  const int *idx, *rowmap, *dcount, *gate;
  int count, rows_pad, pad_ok;
  void *panel, *panel_lo;
  void *npanel;     // candidates: each row's norm column (write_norm_row)
  float *enorm;     // effective norm X2 - 2 mu.x + mu.mu; null: panels and statistics only
  uint32_t *ids;
  unsigned *stats;  // candidates: maxima of the bound (PackStats)
  // queries: the terms of the error bound, the row's largest incoming distance, and the
  // initialisation of its partition roots and of the overflow count
  float4 *qe;
  float *qmx;
  const T *Din;
  int ldD, k, nroots, nproot;  // proot holds nproot rows of nroots
  unsigned *proot;
  int *zero;
};

// Maxima over the candidates (bits of non-negative floats, which order like unsigned integers):
// centred norm |c~|, |effective norm|, norm of the rounding residual |c~ - fmt(c~)|, the scale of
// the FP64 distance's own rounding, and what the norm column leaves of -cn/2 (FP16).
enum PackStats { ST_M = 0, ST_CN, ST_RES, ST_SCALE, ST_NRES, ST_COUNT };
constexpr int STATS_WORDS = 8;

template <typename T>
struct PackArgs {
  // 0 = TF32 (4-byte panel), 1 = BF16, 2 = split BF16 (hi and lo panels), 3 = FP16, scaled by a
  // power of two that takes the sampled coordinates to at most 2^12
  int fmt;
  int d, d_pad;
  PackSide<T> a, b;
  // the shift: from tc_center's partial sums (and written to mu for later launches), or, with part
  // null, read from mu
  const double *part;
  const int *part_n;
  float *mu;
  float *fscale;     // scale of the FP16 format (written and read as mu)
  float kA, kB, kS;  // bound coefficients (TcPlan)
  int *status;
};

template <typename T>
__device__ __forceinline__ void pack_load4(const T *x, int n, bool vec, T (&v)[4]) {
  if (vec) {
    if constexpr (sizeof(T) == 4) {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(x));
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
      const double2 t = __ldg(reinterpret_cast<const double2 *>(x));
      const double2 u = __ldg(reinterpret_cast<const double2 *>(x) + 1);
      v[0] = t.x; v[1] = t.y; v[2] = u.x; v[3] = u.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = j < n ? x[j] : T(0);
  }
}

__device__ __forceinline__ float up_f(float x) { return x; }
__device__ __forceinline__ float up_f(double x) { return __double2float_ru(x); }

// Eight lanes per row, four dimensions per lane at a time: coalesced 16-byte loads of 128 bytes of a
// row, and reductions over eight lanes for four rows at once (a warp per row spent most of its
// instructions on 32-lane FP64 reductions). Candidates and queries of a call share one launch, and
// every block sums the shift from tc_center's partials itself, in one fixed order, instead of
// waiting for a kernel of one block. Bound: HBM reads of the gathered rows.
template <typename T>
__global__ void __launch_bounds__(256) tc_pack(const PackArgs<T> g) {
  extern __shared__ double pack_mu[];  // [d] shift, as doubles
  __shared__ double red[8], redw[8];
  __shared__ unsigned bmx[ST_COUNT];
  const int tid = threadIdx.x, lane = tid & 31, sub = lane & 7;
  if (tid < ST_COUNT) bmx[tid] = 0u;
  int a_rows = g.a.rows_pad, b_rows = g.b.rows_pad;
  if (g.a.gate && *g.a.gate == 0) a_rows = 0;
  if (g.b.gate && *g.b.gate == 0) b_rows = 0;
  int b_count = g.b.count;
  if (g.b.dcount) {
    b_count = *g.b.dcount;
    b_rows = min(b_rows, (b_count + TC_M - 1) / TC_M * TC_M);
  }
  if (blockIdx.x == 0 && tid < 4 && g.b.zero) g.b.zero[tid] = 0;
  if (a_rows + b_rows == 0) return;
  double mu2;
  float fs = 1.0f;
  {
    double s2 = 0.0, wide = 0.0;
    int n = 0;
    if (g.part)
      for (int sl = 0; sl < CENTER_SLICES; sl++) n += g.part_n[sl];
    for (int p = tid; p < g.d; p += 256) {
      float m;
      if (g.part) {
        double tot = 0.0;
        for (int sl = 0; sl < CENTER_SLICES; sl++) tot += g.part[(size_t)sl * g.d + p];
        m = n ? (float)(tot / n) : 0.0f;
        if (blockIdx.x == 0) g.mu[p] = m;
        if (g.fmt == 3) {
          double mn = Num<double>::inf(), mxv = -Num<double>::inf();
          for (int sl = 0; sl < CENTER_SLICES; sl++) {
            mn = fmin(mn, g.part[(size_t)(CENTER_SLICES + sl) * g.d + p]);
            mxv = fmax(mxv, g.part[(size_t)(2 * CENTER_SLICES + sl) * g.d + p]);
          }
          wide = fmax(wide, mxv - mn);
        }
      } else {
        m = g.mu[p];
      }
      pack_mu[p] = (double)m;
      s2 += (double)m * (double)m;
    }
    for (int o = 16; o; o >>= 1) {
      s2 += __shfl_xor_sync(FULL_MASK, s2, o);
      wide = fmax(wide, __shfl_xor_sync(FULL_MASK, wide, o));
    }
    if (lane == 0) {
      red[tid >> 5] = s2;
      redw[tid >> 5] = wide;
    }
    __syncthreads();
    mu2 = 0.0;
    wide = 0.0;
    for (int w = 0; w < 8; w++) {
      mu2 += red[w];
      wide = fmax(wide, redw[w]);
    }
    if (g.fmt == 3) {
      if (g.part) {
        const int e = wide > 0.0 && wide < 1e300 ? 11 - ilogb(wide) : 0;
        fs = ldexpf(1.0f, max(-60, min(60, e)));
        if (blockIdx.x == 0 && tid == 0) *g.fscale = fs;
      } else {
        fs = *g.fscale;
      }
    }
  }
  const double inv_fs = 1.0 / (double)fs;
  unsigned mx[ST_COUNT] = {};
  const int step = gridDim.x * 32;
  // (four rows per warp; a side's rows are whole tiles, so a warp's rows lie on one side)
  for (int r4 = blockIdx.x * 32 + (tid >> 5) * 4; r4 < a_rows + b_rows; r4 += step) {
    const bool is_a = r4 < a_rows;
    const PackSide<T> &s = is_a ? g.a : g.b;
    const int r = (is_a ? r4 : r4 - a_rows) + (lane >> 3);
    const int count = is_a ? s.count : b_count;
    long long row = -1;
    int hr = r;  // heap row (queries)
    if (r < count) {
      if (s.rowmap) hr = s.rowmap[r];
      row = s.idx[hr];
      if (s.pad_ok) hr = (int)row;
      if (s.pad_ok && row == -1) {
        // a padding row of a leaf panel (the batching form): silently empty
      } else if (row < 0 || row >= s.nrows) {
        if (sub == 0) atomicExch(g.status, GSKNN_ERR_INDEX);
        row = -1;
      }
    }
    double s2 = 0.0, smx = 0.0, r2 = 0.0;
    const T *x = s.X + (row >= 0 ? row : 0) * g.d;
    const bool vec = (g.d & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (int p = 4 * sub; p < g.d_pad; p += 32) {
      T v[4] = {T(0), T(0), T(0), T(0)};
      if (row >= 0 && p < g.d) pack_load4<T>(x + p, g.d - p, vec, v);
      float y[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        y[j] = 0.0f;
        if (row >= 0 && p + j < g.d) {
          const double m = pack_mu[p + j], yd = (double)v[j] - m;
          y[j] = (float)yd;
          smx = fma(m, (double)v[j], smx);
          s2 = fma(yd, yd, s2);
        }
      }
      const size_t o = (size_t)r * g.d_pad + p;
      if (g.fmt == 0) {
        uint32_t t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          t[j] = to_tf32(y[j]);
          const double res = (double)(y[j] - __uint_as_float(t[j]));
          r2 = fma(res, res, r2);
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<uint32_t *>(s.panel) + o) =
            make_uint4(t[0], t[1], t[2], t[3]);
      } else if (g.fmt == 3) {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float ys = y[j] * fs;
          const __half v16 = to_f16(ys);
          const double res = (double)(ys - __half2float(v16));
          r2 = fma(res, res, r2);
          h[j] = __half_as_ushort(v16);
        }
        *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(s.panel) + o) =
            make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
      } else {
        uint32_t h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const __nv_bfloat16 hi = __float2bfloat16_rn(y[j]);
          const float rest = y[j] - __bfloat162float(hi);
          h[j] = __bfloat16_as_ushort(hi);
          l[j] = __bfloat16_as_ushort(__float2bfloat16_rn(rest));
          if (g.fmt == 1) r2 = fma((double)rest, (double)rest, r2);
        }
        *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(s.panel) + o) =
            make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        if (g.fmt == 2)
          *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(s.panel_lo) + o) =
              make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
      }
    }
    float qmx = -Num<float>::inf();
    if (s.qmx && row >= 0 && s.Din)
      for (int j = sub; j < s.k; j += 8) qmx = fmaxf(qmx, up_f(s.Din[(size_t)hr * s.ldD + j]));
    if (s.proot && r < s.nproot)
      for (int j = sub; j < s.nroots; j += 8) s.proot[(size_t)r * s.nroots + j] = 0xFFFFFFFFu;
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      s2 += __shfl_xor_sync(FULL_MASK, s2, o);
      smx += __shfl_xor_sync(FULL_MASK, smx, o);
      if (g.fmt != 2) r2 += __shfl_xor_sync(FULL_MASK, r2, o);
      qmx = fmaxf(qmx, __shfl_xor_sync(FULL_MASK, qmx, o));
    }
    if (sub == 0) {
      // |x - mu|^2 expressed through the caller's norm: X2 - 2 mu.x + mu.mu
      const double x2 = row >= 0 ? (double)s.X2[row] : 0.0;
      const float enf = row >= 0 ? (float)(x2 - 2.0 * smx + mu2) : Num<float>::nan();
      float nres = 0.0f;
      if (s.npanel)
        nres = write_norm_row(g.fmt, s.npanel, r, row >= 0,
                              row >= 0 ? -0.5f * enf * (fs * fs) : 0.0f);
      // norms of the centred row and of its rounding residual (in split BF16 a bound on it, 3.2 u^2
      // of the norm, that covers the omitted lo x lo product too), rounded up; and the scale of the
      // FP64 distance's own rounding: the caller's norm, and |x|^2 <= 2 (|x - mu|^2 + |mu|^2)
      const float nrm = row >= 0 ? up_f(sqrt(s2) * (1.0 + 1e-6)) : 0.0f;
      const float res = row < 0 ? 0.0f
                        : g.fmt == 2 ? nrm * (3.2f / 65536.0f)
                                     : up_f(sqrt(r2) * inv_fs * (1.0 + 1e-6));
      const float scale = row >= 0 ? up_f(fmax(fabs(x2), 2.0 * (s2 + mu2))) : 0.0f;
      if (s.enorm) {
        s.enorm[r] = enf;
        if (s.ids) s.ids[r] = row >= 0 ? (uint32_t)row : NO_ID;
      }
      if (s.qe) {
        const float eM = 2.5f * (res + g.kA * nrm) + 2.0f * g.kB * nrm;
        const float eR = g.fmt == 2 ? 0.0f : 2.5f * (nrm + res);
        // (double rows: distances under 1e-30 are left to FP64, floats cannot bound them)
        const float e0 = g.kB * fabsf(enf) + g.kS * scale + (sizeof(T) == 8 ? 1e-30f : 0.0f);
        s.qe[r] = make_float4(eM, eR, e0, 0.0f);
        s.qmx[r] = qmx;
      }
      if (s.stats && row >= 0) {
        mx[ST_M] = max(mx[ST_M], __float_as_uint(nrm));
        mx[ST_CN] = max(mx[ST_CN], __float_as_uint(fabsf(enf) * (1.0f + 1e-6f)));
        mx[ST_RES] = max(mx[ST_RES], __float_as_uint(g.fmt == 2 ? 0.0f : res));
        mx[ST_SCALE] = max(mx[ST_SCALE], __float_as_uint(scale));
        mx[ST_NRES] = max(mx[ST_NRES], __float_as_uint(up_f((double)nres * inv_fs * inv_fs)));
      }
    }
  }
  // the maxima reach the global words once per block (same-address atomics serialize: once per
  // warp took 20 us of a 32,000-row launch)
  unsigned *stats = g.a.stats ? g.a.stats : g.b.stats;
  if (!stats) return;
#pragma unroll
  for (int i = 0; i < ST_COUNT; i++) {
    const unsigned v = __reduce_max_sync(FULL_MASK, mx[i]);
    if (lane == 0 && v) atomicMax(&bmx[i], v);
  }
  __syncthreads();
  if (tid < ST_COUNT && bmx[tid]) atomicMax(&stats[tid], bmx[tid]);
}

// Blocks of a tc_pack launch over `rows` panel rows: 32 rows a block, up to eight blocks per SM,
// grid-stride beyond.
static inline unsigned tc_pack_grid(long long rows) {
  const long long want = (rows + 31) / 32;
  return (unsigned)std::max(1LL, std::min(want, CHIP_SMS * 8LL));
}

// ------------------------------------------------------------------------------------------
// the tensor-core kernel
// ------------------------------------------------------------------------------------------
struct TcParams {
  int Q, nkc, ntiles_r, N, NST, logcap;
  int a_terms;
  int fold;  // norm column in use (set by launch_tc_knn)
  uint32_t idesc;
  const float *cn;
  const float *qn;
  const float4 *qe;       // per-query terms of the error bound (tc_pack)
  const float *qmx;       // largest incoming distance of each query's heap row (-inf: none)
  const unsigned *stats;  // candidate maxima (PackStats)
  float kC, kS;           // bound coefficients of CN and of the distances' own scale
  const float *fscale;    // scale of the FP16 panels (null: 1)
  // Band logs: entry e of a log is a quad, four adjacent columns of the accumulator as the epilogue
  // filtered them (v, or w = -v/2 with the norm column), and the packed position of the first.
  float4 *log;
  uint32_t *logpos;
  int *logcnt;
  // Partition bound. A query's candidates fall into P = NPART * S partitions (split, part). Each
  // keeps a list of the hk = ceil(k / NPART) smallest approximate distances among the quad minima
  // of its own candidates seen so far (each a real candidate of its own), and publishes its root
  // (the list's largest) at proot[query * P + split * NPART + part]
  // (bits of max(root, 0); all bits set while the heap is not full). Any NPART heaps hold at
  // least k real candidates, so the NPART-th smallest root among any partitions of the query --
  // those of its own CTA, and of up to W - 1 other splits as far as they have run -- bounds the
  // query's k-th from above.
  unsigned *proot;
  int hk, W, S;
  float *margin;
  int *status;
  float *dbg;
  long long dbg_ld;
  long long dbg_ncols;
  unsigned long long *counters;  // optional diagnostics (5 counters), may be null
  // optional (escalation pass): the query count on the device (Q is then the capacity and the
  // stride of the per-query arrays) and the heap row of each query
  const int *dQ;
  const int *rowmap;
  // optional (batching form): one entry per CTA -- (query tile, first candidate tile, end
  // candidate tile) -- in place of the (query tile, split) grid; rows whose rowmap entry is -1
  // are padding
  const int4 *qtab;
  // a full log marks the query overflowed at once, without compacting it (a later pass in a
  // narrower format finishes such queries)
  int no_compact;
};

struct SmemLayout {
  uint32_t a_off, b_off, an_off, bn_off, heap_off, ring_off, cn_off, bar_off, tmem_off, total;
};

// Norm column (fold): an all-ones A tile and two slots of candidate norm tiles, 32-byte rows.
constexpr int NORM_ROW = 32;
// Additions of the norm column's MMA (K = 16 in 16-bit formats, 8 in TF32, and the accumulator).
constexpr int NORM_TERMS = 17;

// Partition bound (see TcParams::proot): heap entries per row and part, and the splits whose
// published roots a row reads (its own and up to three more).
__host__ __device__ inline int tc_heap_k(int k) { return (k + NPART - 1) / NPART; }
// Partition lists are kept in whole blocks of LIST_BLOCK values (list_insert). The extreme values
// of the quads a lane has logged but not yet offered to its list wait in a ring in shared memory:
// a warp offers them once any lane has FLUSH_AT (a chunk may add eight), INSERT_BATCH at a time.
constexpr int LIST_BLOCK = 8;
constexpr int LOG_ROOM = 16;  // quads that two chunks of 32 columns may log
constexpr int FLUSH_AT = 6;
constexpr int RING = FLUSH_AT - 1 + 8;
constexpr int INSERT_BATCH = (RING + 1) / 2;
// Where shared memory is short (long query panels, long lists) the tiles may only fit without the
// ring's 13 KB: a flush then reads the quads back from their log, a round trip to L2 for
// INSERT_BATCH of them. Where both fit the ring is up to a quarter faster, also with a stage fewer
// (16,384 x 131,072, d = 64, k = 32 in BF16 2,595 us, without 3,319; 4,000 x 60,000, d = 100, k =
// 100 in split BF16 663 with two stages, without and three 755). Calls that fit only without it
// would else go to the CUDA cores: 4,096 x 60,000, d = 700, k = 32 8,660 us there, 1,068 here.
__host__ __device__ inline int list_slots(int hk) {
  return (hk + LIST_BLOCK - 1) / LIST_BLOCK * LIST_BLOCK;
}
__host__ __device__ inline int tc_window(int S) { return S < 4 ? S : 4; }

// heap_row: heap entries per row over all epilogue parts; ringed: with the ring; fold: the norm
// column areas
__host__ __device__ inline SmemLayout tc_smem_layout(int nkc, int a_terms, int N, int NST,
                                                     int heap_row, bool ringed, bool fold) {
  SmemLayout L;
  uint32_t off = 0;
  L.a_off = off;
  off += (uint32_t)a_terms * nkc * A_CHUNK;
  L.b_off = off;
  off += (uint32_t)NST * N * CHUNK_BYTES;
  L.an_off = off;  // 1024-aligned: every area above is a multiple of 1 KB
  off += fold ? (uint32_t)TC_M * NORM_ROW : 0u;
  L.bn_off = off;
  off += fold ? 2u * N * NORM_ROW : 0u;
  L.heap_off = off;
  off += (uint32_t)heap_row * TC_M * 4;
  L.ring_off = off;
  off += ringed ? (uint32_t)NPART * RING * TC_M * 4 : 0u;
  off = (off + 15) & ~15u;
  L.cn_off = off;  // candidate norms of the tiles in flight, copied by the MMA warp
  off += fold ? 0u : (uint32_t)CN_SLOTS * N * 4;
  off = (off + 7) & ~7u;
  L.bar_off = off;
  // full, empty, tfull[2], tempty[2], afull, cnfull, nfull[2], nempty[2]
  off += (uint32_t)(2 * NST + 9 + CN_SLOTS) * 8;
  L.tmem_off = off;
  off += 16;
  L.total = off + 1024;  // alignment slack
  return L;
}

struct EpiState {
  // root: this part's heap root; o1 <= o2: the two smallest roots among the other partitions
  // the row reads (as last published); pub: what this part last published
  // Tv: the filter bound on v = d' - qn'; Tw = -Tv/2 the same bound on w = -v/2 (norm column)
  // (FP16: w in the panels' scale s, Tw = -Tv s^2 / 2, v = -2 w / s^2)
  float qn, E2, thr0, root, o1, o2, pub, thr, Tv, Tw;
  float vw, wv;  // v = vw * w, w = wv * v: powers of two
  int cnt;   // logged quads
  int done;  // of them, already offered to the heap
  int ovf;
  // optional diagnostics: flushes, chunks that took the slow path
  unsigned n_fl, n_sc;
};

// Any two partitions' heaps hold at least k real candidates, so the second smallest root among
// this part's and the others' bounds the query's k-th smallest approximate distance from above.
__device__ __forceinline__ void refresh_threshold(EpiState &s) {
  static_assert(NPART == 2, "the bound takes the NPART-th smallest root");
  // (exact distances are clamped at 0: a k-th bound below it admits every clamped candidate too)
  float t = fmaxf(fminf(fmaxf(s.root, s.o1), s.o2), 0.0f) + s.E2;
  s.thr = t < s.thr0 ? t : s.thr0;
  // padding rows past the last query never admit; nor does a row whose log overflowed (the
  // query is finished by a later pass), so its chunks stop taking the slow path
  if (s.thr == -Num<float>::inf() || s.ovf) {
    s.Tv = -Num<float>::inf();
    s.Tw = Num<float>::inf();
    return;
  }
  // filter in the v = d' - qn' space with slack for the rounding of the subtraction
  s.Tv = (s.thr - s.qn) + (fabsf(s.thr) + fabsf(s.qn)) * 2.4e-7f + 1e-30f;
  s.Tw = s.wv * s.Tv;  // exact: v <= Tv  <=>  w >= Tw
}

// Partition lists: every row and part keeps its hk smallest values ascending in shared memory,
// element i of this thread's row at list[i * TC_M + row] (bank-conflict free across a warp), hk
// rounded up to whole blocks of LIST_BLOCK. The "root" is element hk - 1. A batch of values goes
// through one block of registers after the other: with a sorted block a, inserting x gives
// a'[i] = min(max(a[i-1], x), a[i]) for every i at once, and the block's largest moves on to the
// next block. A binary heap's sift-down is a chain of shared-memory round trips per value (7,700
// cycles a flush at hk = 16); this is arithmetic without one.
template <int NB>
__device__ __forceinline__ void list_insert(float *list, int row, int hk, float (&x)[NB]) {
  for (int b = 0; b < hk; b += LIST_BLOCK) {
    float a[LIST_BLOCK];
    float *const blk = list + b * TC_M + row;
#pragma unroll
    for (int i = 0; i < LIST_BLOCK; i++) a[i] = blk[i * TC_M];
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const float v = x[j];
      x[j] = fmaxf(a[LIST_BLOCK - 1], v);  // moves on to the next block
#pragma unroll
      for (int i = LIST_BLOCK - 1; i > 0; i--) a[i] = fminf(fmaxf(a[i - 1], v), a[i]);
      a[0] = fminf(a[0], v);
    }
#pragma unroll
    for (int i = 0; i < LIST_BLOCK; i++) blk[i * TC_M] = a[i];
  }
}

// Whether the extreme value of a quad or chunk (largest w with the norm column, else smallest v)
// admits it under the row's filter bound.
template <bool FOLD>
__device__ __forceinline__ bool epi_hit(const EpiState &s, float m) {
  return FOLD ? m >= s.Tw : m <= s.Tv;
}
template <bool FOLD>
__device__ __forceinline__ float quad_extreme(float a, float b, float c, float d) {
  return FOLD ? fmaxf(fmax3(a, b, c), d) : fminf(fmin3(a, b, c), d);
}
// approximate distance d' of a filtered value: v + qn, with v = -2w (exact)
template <bool FOLD>
__device__ __forceinline__ float epi_dist(const EpiState &s, float x) {
  return FOLD ? fmaf(s.vw, x, s.qn) : x + s.qn;
}

// Publish the list's root to the other partitions and tighten the threshold.
__device__ __forceinline__ void epi_publish(EpiState &s, const float *heap, int row, int hk,
                                            unsigned *pslot) {
  s.root = heap[(hk - 1) * TC_M + row];
  // published as non-negative float bits (a larger value bounds as well), which order like
  // unsigned integers; only this partition writes its slot
  const float pv = fmaxf(s.root, 0.0f);
  if (pv < s.pub) {
    __stcg(pslot, __float_as_uint(pv));
    s.pub = pv;
  }
  refresh_threshold(s);
}

// Offer a chunk's eight quads to the row's list, by their extreme values.
template <bool FOLD>
__device__ __forceinline__ void epi_offer(const EpiState &s, float *heap, int row, int hk,
                                          const float (&g)[8]) {
  float x[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    x[j] = epi_dist<FOLD>(s, g[j]);
    // padding columns; and padding rows, whose published root would be query 0's
    if (!(x[j] < Num<float>::inf()) || s.thr0 == -Num<float>::inf()) x[j] = Num<float>::inf();
  }
  list_insert(heap, row, hk, x);
}

// Offer the quads logged since the last flush to the row's list, by their extreme values in the
// ring (all lanes of the warp together), publish the new root to the other partitions and tighten
// the threshold. Without a ring the quads are read back from their log, `lg`.
template <bool FOLD, bool RINGED>
__device__ __forceinline__ void epi_flush(EpiState &s, float *heap, const float *ring,
                                          const float4 *lg, int row, int hk, unsigned *pslot) {
  s.n_fl++;
  const int np = s.cnt - s.done;
  for (int e = 0; __any_sync(FULL_MASK, e < np); e += INSERT_BATCH) {
    float x[INSERT_BATCH];
#pragma unroll
    for (int j = 0; j < INSERT_BATCH; j++) {
      x[j] = Num<float>::inf();
      if (e + j < np) {
        if constexpr (RINGED) {
          x[j] = epi_dist<FOLD>(s, ring[(e + j) * TC_M + row]);
        } else {
          const float4 v = __ldcg(lg + s.done + e + j);
          x[j] = epi_dist<FOLD>(s, quad_extreme<FOLD>(v.x, v.y, v.z, v.w));
        }
      }
    }
    list_insert(heap, row, hk, x);
  }
  s.done = s.cnt;
  epi_publish(s, heap, row, hk, pslot);
}

// Drops the entries above the current threshold (the filter bound Tw or Tv) from the logs of the
// lanes that `want` it, all of them already offered to the lists; returns the lane's new count. The
// warp takes one log after the other, 32 entries at a time with coalesced loads. One lane per log, an
// entry at a time, is a chain of round trips to L2 while the tile's other rows wait: 17.2 M
// cycles a CTA on 16,384 x 60,000, d = 80, k = 32 in split BF16 on clusters of sigma 0.01, 2.65 M so.
template <bool FOLD>
__device__ __noinline__ int log_compact(float4 *lg, uint32_t *lp, int cnt, float bound, bool want) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the logs' stores before the other lanes' loads
  for (unsigned m = __ballot_sync(FULL_MASK, want); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    float4 *const l = reinterpret_cast<float4 *>(
        __shfl_sync(FULL_MASK, reinterpret_cast<unsigned long long>(lg), src));
    uint32_t *const p = reinterpret_cast<uint32_t *>(
        __shfl_sync(FULL_MASK, reinterpret_cast<unsigned long long>(lp), src));
    const int n = __shfl_sync(FULL_MASK, cnt, src);
    const float bnd = __shfl_sync(FULL_MASK, bound, src);
    int w = 0;
    for (int e = 0; e < n; e += 32) {
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      uint32_t pos = 0u;
      const bool in = e + lane < n;
      if (in) {
        v = __ldcg(l + e + lane);
        pos = __ldcg(p + e + lane);
      }
      const float x = quad_extreme<FOLD>(v.x, v.y, v.z, v.w);
      const bool keep = in && (FOLD ? x >= bnd : x <= bnd);
      const unsigned k = __ballot_sync(FULL_MASK, keep);
      __syncwarp();  // all of the step's loads before its stores, which may reach their places
      if (keep) {
        const int at = w + __popc(k & ((1u << lane) - 1u));
        l[at] = v;
        p[at] = pos;
      }
      w += __popc(k);
    }
    if (lane == src) cnt = w;
  }
  __syncwarp();
  return cnt;
}

// FOLD: the candidate norms enter through the MMA (the norm column, write_norm_row), so the
// accumulator holds w = -v/2 and the epilogue filters it directly; else the epilogue forms
// v = cn - 2<q~, c~> from the norms it reads into shared memory.
template <int FMT, bool FOLD, bool RINGED>
__global__ void __launch_bounds__(NTHREADS, 1)
    tc_knn(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tAlo,
           const __grid_constant__ CUtensorMap tB, const __grid_constant__ CUtensorMap tBlo,
           const __grid_constant__ CUtensorMap tBn, const TcParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int TERMS = FMT == 2 ? 2 : 1;  // B tiles per K chunk
  // escalation pass: launched for the largest possible query count, the tiles past the count
  // on the device exit before any set-up
  const int Qn = p.dQ ? *p.dQ : p.Q;
  // grid: (query tile, split), query tiles fastest, so that a query's later splits mostly start
  // after its first ones finished and take their final roots as a tight bound from the first
  // tile; or one block per qtab entry
  if (!p.qtab && (int)blockIdx.x * TC_M >= Qn) return;
  const uint32_t raw = su32(smem_raw);
  unsigned char *smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  const SmemLayout L =
      tc_smem_layout(p.nkc, p.a_terms, p.N, p.NST, NPART * list_slots(p.hk), RINGED,
                     FOLD);
  unsigned char *sA = smem + L.a_off;
  unsigned char *sB = smem + L.b_off;
  unsigned char *sAn = smem + L.an_off;
  unsigned char *sBn = smem + L.bn_off;
  float *heap = reinterpret_cast<float *>(smem + L.heap_off);
  float *ring = reinterpret_cast<float *>(smem + L.ring_off);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar_off);
  uint64_t *full = bars;
  uint64_t *empty = bars + p.NST;
  uint64_t *tfull = bars + 2 * p.NST;
  uint64_t *tempty = bars + 2 * p.NST + 2;
  uint64_t *afull = bars + 2 * p.NST + 4;
  uint64_t *cnfull = bars + 2 * p.NST + 5;
  uint64_t *nfull = cnfull + CN_SLOTS;  // norm tile of slot b landed
  uint64_t *nempty = nfull + 2;         // norm tile of slot b read by the tile's MMAs
  float *cn_s = reinterpret_cast<float *>(smem + L.cn_off);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + L.tmem_off);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int qt = blockIdx.x, t_begin, t_end;
  const int split = blockIdx.y;
  if (p.qtab) {
    const int4 w = p.qtab[blockIdx.x];
    qt = w.x;
    t_begin = w.y;
    t_end = w.z;
  } else {
    // balanced ranges: every split gets floor or ceil of ntiles_r / S tiles
    t_begin = (int)((long long)split * p.ntiles_r / p.S);
    t_end = (int)((long long)(split + 1) * p.ntiles_r / p.S);
  }
  if (t_end > p.ntiles_r) t_end = p.ntiles_r;
  const int ntile = t_end > t_begin ? t_end - t_begin : 0;
  const int N = p.N;
  const uint32_t b_stage_bytes = (uint32_t)N * CHUNK_BYTES;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], NEPI);
    }
    mbar_init(afull, 1);
    for (int c = 0; c < CN_SLOTS; c++) mbar_init(&cnfull[c], 1);
    for (int b = 0; b < 2; b++) {
      mbar_init(&nfull[b], 1);
      mbar_init(&nempty[b], 1);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, (uint32_t)(2 * N));
    tmem_relinquish();
  }
  // the per-row heaps start at +inf before any epilogue warp reads a root (each part of a lane
  // quarter reads the other's root as part of its bound)
  for (int i = threadIdx.x; i < NPART * list_slots(p.hk) * TC_M; i += NTHREADS)
    heap[i] = Num<float>::inf();
  if (FOLD) {
    // the all-ones A side of the norm column (every 16-byte chunk alike, so any swizzle of it is
    // the same bytes), made visible to the tensor core's operand reads
    // (FP16: the weights 2^14, 2^3, 2^-8, then zeros)
    const uint32_t one = FMT == 0 ? 0x3F800000u : 0x3F803F80u;
    uint32_t *an = reinterpret_cast<uint32_t *>(sAn);
    for (int i = threadIdx.x; i < TC_M * NORM_ROW / 4; i += NTHREADS)
      an[i] = FMT != 1 || !p.fscale ? one
              : (i & 3) == 0        ? 0x48007400u
              : (i & 3) == 1        ? 0x00001C00u
                                    : 0u;
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  bool failed = false;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0 && ntile > 0) {
      prefetch_tmap(&tA);
      prefetch_tmap(&tB);
      const int celems = FMT == 0 ? 32 : 64;
      mbar_expect_tx(afull, (uint32_t)(p.a_terms * p.nkc * A_CHUNK));
      for (int kc = 0; kc < p.nkc; kc++) {
        tma_load_2d(sA + kc * A_CHUNK, &tA, kc * celems, qt * TC_M, afull);
        if (FMT == 2)
          tma_load_2d(sA + (p.nkc + kc) * A_CHUNK, &tAlo, kc * celems, qt * TC_M, afull);
      }
      int stage = 0;
      uint32_t round = 0;  // parity of the stage's use
      if (FOLD) prefetch_tmap(&tBn);
      for (int lt = 0; lt < ntile && !failed; lt++) {
        const int tile = t_begin + lt;
        if (FOLD) {
          // the tile's norm column, into slot lt & 1 once the MMAs of tile lt - 2 read it
          const int nb = lt & 1;
          if (!mbar_wait(&nempty[nb], ((uint32_t)(lt >> 1) & 1u) ^ 1u)) { failed = true; break; }
          mbar_expect_tx(&nfull[nb], (uint32_t)(N * NORM_ROW));
          tma_load_2d(sBn + (uint32_t)nb * N * NORM_ROW, &tBn, 0, tile * N, &nfull[nb]);
        }
        // a stage is one K chunk of one term: in split BF16 the hi and lo tiles take stages in
        // turn, which the pipeline refills one by one
        for (int i = 0; i < TERMS * p.nkc; i++) {
          const int s = stage;
          if (!mbar_wait(&empty[s], round ^ 1u)) { failed = true; break; }
          if (++stage == p.NST) { stage = 0; round ^= 1u; }
          mbar_expect_tx(&full[s], b_stage_bytes);
          tma_load_2d(sB + (uint32_t)s * b_stage_bytes, i % TERMS ? &tBlo : &tB,
                      i / TERMS * celems, tile * N, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0 && ntile > 0) {
      const long long t_start = p.counters ? clock64() : 0;
      long long w_tempty = 0, w_full = 0;
      if (!mbar_wait(afull, 0)) failed = true;
      tc_fence_after();
      const uint32_t a_base = su32(sA), b_base = su32(sB);
      int stage = 0;
      uint32_t round = 0;  // parity of the stage's use
      for (int lt = 0; lt < ntile && !failed; lt++) {
        const int b = lt & 1;
        const uint32_t use = (uint32_t)(lt >> 1);
        long long t0 = p.counters ? clock64() : 0;
        if (!mbar_wait(&tempty[b], (use & 1u) ^ 1u)) { failed = true; break; }
        if (p.counters) w_tempty += clock64() - t0;
        // every epilogue warp has released tile lt - 2, so all of them are done with tile lt - 3
        // and its norm slot: fetch this tile's candidate norms there
        const uint32_t tmem_d = tmem_base + (uint32_t)(b * N);
        if (!FOLD) {
          const int c = lt % CN_SLOTS;
          mbar_expect_tx(&cnfull[c], (uint32_t)(N * 4));
          bulk_g2s(cn_s + c * N, p.cn + (size_t)(t_begin + lt) * N, (uint32_t)(N * 4),
                   &cnfull[c]);
        }
        tc_fence_after();
        // The norm column's MMA. In split BF16 it goes last: first, every later addition would add a
        // rounding of |cn|/2 to the bound (E at d = 80 and 128 was 1.27 times what it is without the
        // column, and clusters overflowed their logs). The single-term formats' bound is their input
        // rounding, and last it stands behind the tile's final stage: 32,768 x 262,144, d = 256, k = 64
        // in FP16 5,502 us, first 5,424.
        auto norm_mma = [&](uint32_t accumulate) {
          if (!mbar_wait(&nfull[b], use & 1u)) { failed = true; return; }
          tc_fence_after();
          const uint64_t ad = sdesc_k_sw32(su32(sAn));
          const uint64_t bd = sdesc_k_sw32(su32(sBn) + (uint32_t)b * N * NORM_ROW);
          if (FMT == 0) mma_tf32(tmem_d, ad, bd, p.idesc, accumulate);
          else mma_f16(tmem_d, ad, bd, p.idesc, accumulate);
        };
        constexpr bool NORM_FIRST = FOLD && FMT != 2;
        if (NORM_FIRST) {
          norm_mma(0u);
          if (failed) break;
        }
        for (int i = 0; i < TERMS * p.nkc; i++) {
          const int s = stage, kc = i / TERMS;
          const bool lo = i % TERMS != 0;
          t0 = p.counters ? clock64() : 0;
          if (!mbar_wait(&full[s], round)) { failed = true; break; }
          if (++stage == p.NST) { stage = 0; round ^= 1u; }
          if (p.counters) w_full += clock64() - t0;
          tc_fence_after();
          // One thread issues all of a CTA's MMAs and, with short ones, its own instructions set the
          // pace: a division for the stage and descriptors built from scratch for each MMA took
          // 4.17 M cycles a CTA on 32,768 x 262,144, d = 256, k = 64 in split BF16 (128-column
          // tiles) and 16.95 ms a call, this 13.58 ms; TF32 there 14.2 -> 11.4 ms; 65,536 x
          // 262,144, d = 64, k = 32 6.40 -> 5.93 ms. K steps of 32 bytes: two more in a
          // descriptor's address field (16-byte units).
          const uint64_t ad = sdesc_k_sw128(a_base + (uint32_t)kc * A_CHUNK);
          const uint64_t bd = sdesc_k_sw128(b_base + (uint32_t)s * b_stage_bytes);
          const uint32_t first = NORM_FIRST || i != 0 ? 1u : 0u;
          if (FMT == 2 && !lo) {
            // hi stage: the query's lo part too
            const uint64_t ld = sdesc_k_sw128(a_base + (uint32_t)(p.nkc + kc) * A_CHUNK);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              mma_f16(tmem_d, ad + 2u * ks, bd + 2u * ks, p.idesc, ks == 0 ? first : 1u);
              mma_f16(tmem_d, ld + 2u * ks, bd + 2u * ks, p.idesc, 1u);
            }
          } else {
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
              if (FMT == 0)
                mma_tf32(tmem_d, ad + 2u * ks, bd + 2u * ks, p.idesc, ks == 0 ? first : 1u);
              else
                mma_f16(tmem_d, ad + 2u * ks, bd + 2u * ks, p.idesc, ks == 0 ? first : 1u);
            }
          }
          mma_commit(&empty[s]);
        }
        if (FOLD && !NORM_FIRST && !failed) norm_mma(1u);
        if (!failed) {
          if (FOLD) mma_commit(&nempty[b]);
          mma_commit(&tfull[b]);
        }
      }
      if (p.counters) {
        atomicAdd(&p.counters[7], (unsigned long long)w_full);
        atomicAdd(&p.counters[8], (unsigned long long)w_tempty);
        atomicAdd(&p.counters[10], (unsigned long long)(clock64() - t_start));
      }
    }
  } else {
    // ---------------- epilogue: one query row per thread ----------------
    const int lq = warp & 3;            // TMEM lane quarter this warp may access
    const int part = (warp - 2) >> 2;   // column range of the tile (and heap) of this warp
    const int row = lq * 32 + lane;
    const int gq = qt * TC_M + row;
    const bool valid = gq < Qn && (!p.rowmap || p.rowmap[gq] >= 0);
    float *const myheap = heap + part * list_slots(p.hk) * TC_M;
    const float *const otherheap = heap + (NPART - 1 - part) * list_slots(p.hk) * TC_M;
    float *const myring = ring + part * RING * TC_M;
    const int P = NPART * p.S;  // partitions of a query
    EpiState s;
    s.cnt = 0;
    s.done = 0;
    s.ovf = 0;
    s.o1 = Num<float>::inf();
    s.o2 = Num<float>::inf();
    s.pub = Num<float>::inf();
    s.n_fl = s.n_sc = 0;
    unsigned *const pslot = p.proot + (size_t)(valid ? gq : 0) * P + NPART * split + part;
    const unsigned *const prow = p.proot + (size_t)(valid ? gq : 0) * P;
    {
      const float fs = FMT == 1 && p.fscale ? *p.fscale : 1.0f;
      s.wv = -0.5f * (fs * fs);
      s.vw = 1.0f / s.wv;
    }
    s.root = Num<float>::inf();
    s.qn = 0.0f;
    s.E2 = 0.0f;
    s.thr0 = Num<float>::inf();
    if (valid) {
      s.qn = p.qn[gq];
      const float4 e = p.qe[gq];
      const float E = e.x * __uint_as_float(p.stats[ST_M]) +
                      e.y * __uint_as_float(p.stats[ST_RES]) + e.z +
                      p.kC * __uint_as_float(p.stats[ST_CN]) +
                      p.kS * __uint_as_float(p.stats[ST_SCALE]) +
                      (FOLD ? 2.5f * __uint_as_float(p.stats[ST_NRES]) : 0.0f);
      s.E2 = 2.0f * E;
      const float mx = p.qmx[gq];
      if (mx > -Num<float>::inf()) s.thr0 = mx + s.E2;
      refresh_threshold(s);
      if (split == 0 && part == 0) p.margin[gq] = s.E2;
    } else {
      // padding row: its log and shared-bound pointers alias query 0, so it must never admit a
      // candidate; the -inf ceiling survives every threshold refresh
      s.thr0 = -Num<float>::inf();
      s.thr = -Num<float>::inf();
      s.Tv = -Num<float>::inf();
      s.Tw = Num<float>::inf();
    }
    const int lslot = NPART * split + part;  // this warp's log among the NPART*S logs of the query
    float4 *const lg = p.log + ((size_t)lslot * p.Q + (valid ? gq : 0)) * p.logcap;
    uint32_t *const lp = p.logpos + ((size_t)lslot * p.Q + (valid ? gq : 0)) * p.logcap;
    // Fast part of a 32-column chunk: v = d' - qn' over the accumulator values in place (with the
    // norm column the registers already hold w = -v/2), the extreme value of every quad of four
    // columns and of the chunk, in three-input steps. Two chunks' fast parts run back to back in
    // one basic block so their independent arithmetic overlaps.
    auto fast = [&](uint32_t (&r)[32], float (&g)[8], const float *cnt, int c0) -> float {
      if constexpr (!FOLD) {
        const float4 *cn4 = reinterpret_cast<const float4 *>(cnt + c0);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float4 c4 = cn4[j];
          float v0, v1, v2, v3;
          fma2(v0, v1, __uint_as_float(r[4 * j + 0]), __uint_as_float(r[4 * j + 1]), s.vw, c4.x,
               c4.y);
          fma2(v2, v3, __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]), s.vw, c4.z,
               c4.w);
          r[4 * j + 0] = __float_as_uint(v0);
          r[4 * j + 1] = __float_as_uint(v1);
          r[4 * j + 2] = __float_as_uint(v2);
          r[4 * j + 3] = __float_as_uint(v3);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; j++)
        g[j] = quad_extreme<FOLD>(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                  __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
      if constexpr (FOLD)
        return fmax3(fmax3(g[0], g[1], g[2]), fmax3(g[3], g[4], g[5]), fmaxf(g[6], g[7]));
      else
        return fmin3(fmin3(g[0], g[1], g[2]), fmin3(g[3], g[4], g[5]), fminf(g[6], g[7]));
    };
    // whether a chunk's extreme value admits it
    auto hit = [&](float m) { return epi_hit<FOLD>(s, m); };
    auto dbg_write = [&](const uint32_t (&r)[32], size_t cbase, int c0) {
      for (int i = 0; i < 32; i++) {
        const long long col = (long long)cbase + c0 + i;
        const float v = FOLD ? s.vw * __uint_as_float(r[i]) : __uint_as_float(r[i]);
        if (col < p.dbg_ncols) p.dbg[(size_t)gq * p.dbg_ld + col] = v + s.qn;
      }
    };
    // Slow part, for a chunk in which some lane has a candidate under its threshold: every lane
    // logs its quads that have one, whole (four registers that lie side by side, one 16-byte store
    // and one 4-byte store, both predicated; no value is selected by index and no loop runs over
    // the survivors). What it costs is the eight predicated stores' issue; logging single
    // candidates, each found by a mask and selected by a 31-instruction tree, took about 1,150
    // cycles a chunk, this about 250. With the partition lists in registers during a flush and the
    // other splits' roots first touched a tile after their loads: tc_knn on 65,536 x 262,144,
    // d = 64, k = 32 8,283 -> 5,853 us; 32,768 x 262,144, d = 256, k = 64 6,790 -> 4,466 us;
    // 2,003 x 30,011, d = 20 105 -> 64 us; 16 x 4,096 42 -> 10 us; 8 trees over 262,144 points
    // 6.1 -> 3.1 ms.
    auto slow = [&](const uint32_t (&r)[32], const float (&g)[8], uint32_t pos, bool offered) {
      s.n_sc++;
      const uint32_t rbase = su32(myring + row);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float4 *const at = lg + s.cnt;
        const uint32_t *const pt = lp + s.cnt;
        const uint32_t rp = rbase + (uint32_t)(s.cnt - s.done) * (TC_M * 4);
        if constexpr (FOLD)
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ge.f32 p, %1, %2;\n\t"
              "@p st.global.v4.b32 [%3], {%4, %5, %6, %7};\n\t"
              "@p st.global.b32 [%8], %9;\n\t"
              "@p st.shared.f32 [%10], %1;\n\t"
              "@p add.s32 %0, %0, 1;\n\t}\n"
              : "+r"(s.cnt)
              : "f"(g[j]), "f"(s.Tw), "l"(at), "r"(r[4 * j]), "r"(r[4 * j + 1]),
                "r"(r[4 * j + 2]), "r"(r[4 * j + 3]), "l"(pt), "r"(pos + 4 * j), "r"(rp)
              : "memory");
        else if constexpr (RINGED)
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.le.f32 p, %1, %2;\n\t"
              "@p st.global.v4.b32 [%3], {%4, %5, %6, %7};\n\t"
              "@p st.global.b32 [%8], %9;\n\t"
              "@p st.shared.f32 [%10], %1;\n\t"
              "@p add.s32 %0, %0, 1;\n\t}\n"
              : "+r"(s.cnt)
              : "f"(g[j]), "f"(s.Tv), "l"(at), "r"(r[4 * j]), "r"(r[4 * j + 1]),
                "r"(r[4 * j + 2]), "r"(r[4 * j + 3]), "l"(pt), "r"(pos + 4 * j), "r"(rp)
              : "memory");
        else
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.le.f32 p, %1, %2;\n\t"
              "@p st.global.v4.b32 [%3], {%4, %5, %6, %7};\n\t"
              "@p st.global.b32 [%8], %9;\n\t"
              "@p add.s32 %0, %0, 1;\n\t}\n"
              : "+r"(s.cnt)
              : "f"(g[j]), "f"(s.Tv), "l"(at), "r"(r[4 * j]), "r"(r[4 * j + 1]),
                "r"(r[4 * j + 2]), "r"(r[4 * j + 3]), "l"(pt), "r"(pos + 4 * j)
              : "memory");
      }
      if (offered) s.done = s.cnt;  // the lists have these already
      if (__any_sync(FULL_MASK, s.cnt - s.done >= FLUSH_AT))
        epi_flush<FOLD, RINGED>(s, myheap, myring, lg, row, p.hk, pslot);
    };
    // Logs without room for another two chunks drop what has left the band. Called between chunks,
    // when no accumulator values are held: the call's registers would else be spilled around it,
    // 1.2 times the ordinary pass's time. A compaction that frees less than a quarter of the log
    // marks it overflowed: repeated ones that each free a few entries would cost a full read of the
    // log per chunk. (Half, as when an entry was read at a time, gives up logs that would have
    // lasted: 8,192 x 250,000, d = 32, k = 128 on clusters of sigma 0.01 3,121 brute-forced queries
    // and 118 ms, now 246 and 16 ms.)
    auto make_room = [&]() {
      const bool full = s.cnt > p.logcap - LOG_ROOM && !s.ovf;
      if (!__any_sync(FULL_MASK, full)) return;
      epi_flush<FOLD, RINGED>(s, myheap, myring, lg, row, p.hk, pslot);
      if (!p.no_compact) {
        const int left = log_compact<FOLD>(lg, lp, s.cnt, FOLD ? s.Tw : s.Tv, full);
        if (full) s.cnt = s.done = left;
      }
      if (full && s.cnt > min(p.logcap / 4 * 3, p.logcap - LOG_ROOM)) {
        s.ovf = 1;
        refresh_threshold(s);
      }
    };
    // the roots up to three other splits have published (all bits set, which orders last: a list
    // not full yet). The loads for the next tile are issued a tile ahead and their values are
    // first touched there, so that their latency hides behind the tile's work
    uint2 win[3];
    auto load_window = [&]() {
#pragma unroll
      for (int w = 0; w < 3; w++) {
        win[w] = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);
        if (w + 1 < p.W) {
          int sp = split + w + 1;
          if (sp >= p.S) sp -= p.S;
          win[w] = __ldcg(reinterpret_cast<const uint2 *>(prow + NPART * sp));
        }
      }
    };
    // their two smallest
    auto read_window = [&](unsigned &m1, unsigned &m2) {
      m1 = m2 = 0xFFFFFFFFu;
#pragma unroll
      for (int w = 0; w < 3; w++) {
        m2 = min(m2, max(m1, win[w].x));
        m1 = min(m1, win[w].x);
        m2 = min(m2, max(m1, win[w].y));
        m1 = min(m1, win[w].y);
      }
    };
    auto as_bound = [](unsigned u) {
      return u == 0xFFFFFFFFu ? Num<float>::inf() : __uint_as_float(u);
    };
    load_window();
    // the other part of this lane quarter (same rows, other columns) keeps its list in shared
    // memory: its root is read directly (one 4-byte word, written whole)
    auto other_root = [&]() {
      return *reinterpret_cast<volatile const float *>(&otherheap[(p.hk - 1) * TC_M + row]);
    };
    // the two smallest roots among the other partitions, and the threshold they give
    auto look_around = [&]() {
      unsigned win1, win2;
      read_window(win1, win2);
      const float a = other_root(), w1 = as_bound(win1), w2 = as_bound(win2);
      const float o1 = fminf(a, w1), o2 = fminf(fmaxf(a, w1), w2);
      if (o1 < s.o1 || o2 < s.o2) {
        s.o1 = fminf(s.o1, o1);
        s.o2 = fminf(s.o2, o2);
        refresh_threshold(s);
      }
    };
    // rows with no bound yet, and lists that the first tile's quads fill
    bool first = p.hk <= N / NPART / 4 &&
                 __any_sync(FULL_MASK, valid && !(s.thr0 < Num<float>::inf()));
    const long long t_start = p.counters ? clock64() : 0;
    long long w_tfull = 0;
    for (int lt = 0; lt < ntile && !failed; lt++) {
      const int b = lt & 1, c = lt % CN_SLOTS;
      const uint32_t use = (uint32_t)(lt >> 1), cuse = (uint32_t)(lt / CN_SLOTS);
      // (every tile while the bound still falls fast, then every fourth: the update takes about
      // 420 of a tile's 3,000 cycles)
      const bool look = lt < 16 || (lt & 3) == 0;
      if (valid && look) look_around();
      if (look) load_window();
      const long long t0 = p.counters ? clock64() : 0;
      if (!mbar_wait(&tfull[b], use & 1u)) { failed = true; break; }
      if (!FOLD && !mbar_wait(&cnfull[c], cuse & 1u)) { failed = true; break; }
      if (p.counters) w_tfull += clock64() - t0;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(b * N);
      const float *cnt = cn_s + c * N;
      const int tile = t_begin + lt;
      const size_t cbase = (size_t)tile * N;
      // this warp's N/NPART columns, 64 at a time (two 32-column chunks per TMEM wait); the
      // accumulator is freed for the MMA warp once the tile's last loads of every epilogue warp
      // have landed (the norms stay in their own slot)
      const int cb = part * (N / NPART), ce = cb + N / NPART;
      if (!p.dbg && __all_sync(FULL_MASK, !valid || s.ovf)) {
        // every row of this warp is padding or finished by a later pass: release the
        // accumulator without reading it (after its tile landed, so the release counts for
        // this tile)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[b]);
        continue;
      }
      // The first tile of rows without an incoming bound is read twice: once to offer its quads'
      // extreme values to the lists, then to log what lies under the bound that gives. Logging as
      // the lists fill took most of a short split's time: every lane stores every quad, 32 lines
      // per store (2,003 x 30,011, d = 20, nine splits: 882 -> 395 quads a query, 66 -> 54 us).
      const bool warm = first;
      if (warm) {
        first = false;
        for (int c0 = cb; c0 < ce; c0 += 32) {
          uint32_t ra[32];
          __syncwarp();
          tmem_ld32(taddr + (uint32_t)c0, ra);
          tmem_wait_ld();
          reg_fence32(ra);
          float ga[8];
          fast(ra, ga, cnt, c0);
          epi_offer<FOLD>(s, myheap, row, p.hk, ga);
        }
        epi_publish(s, myheap, row, p.hk, pslot);
        // the other part fills its list at the same time: give it a moment
        for (int i = 0; i < 64; i++) {
          const bool there = other_root() < Num<float>::inf();
          if (__all_sync(FULL_MASK, !valid || there)) break;
          __nanosleep(32);
        }
        if (valid) look_around();
      }
      for (int c0 = cb; c0 < ce; c0 += 64) {
        uint32_t ra[32], rb[32];
        __syncwarp();
        tmem_ld32(taddr + (uint32_t)c0, ra);
        tmem_ld32(taddr + (uint32_t)c0 + 32u, rb);
        tmem_wait_ld();
        reg_fence32(ra);
        reg_fence32(rb);
        if (c0 + 64 >= ce) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[b]);
        }
        float ga[8], gb[8];
        const float ma = fast(ra, ga, cnt, c0);
        const float mb = fast(rb, gb, cnt, c0 + 32);
        if (p.dbg && valid) {
          dbg_write(ra, cbase, c0);
          dbg_write(rb, cbase, c0 + 32);
        }
        const bool ha = __any_sync(FULL_MASK, hit(ma));
        if (ha) slow(ra, ga, (uint32_t)(cbase + c0), warm);
        const bool hb = __any_sync(FULL_MASK, hit(mb));
        if (hb) slow(rb, gb, (uint32_t)(cbase + c0 + 32), warm);
        if (ha || hb) make_room();
      }
    }
    epi_flush<FOLD, RINGED>(s, myheap, myring, lg, row, p.hk, pslot);
    if (valid) p.logcnt[(size_t)lslot * p.Q + gq] = s.cnt | (s.ovf ? (int)LOG_OVF : 0);
    if (p.counters) {
      atomicAdd(&p.counters[0], (unsigned long long)s.cnt);
      if (lane == 0) {
        atomicAdd(&p.counters[2], (unsigned long long)s.n_fl);
        atomicAdd(&p.counters[3], (unsigned long long)s.n_sc);
        atomicAdd(&p.counters[4], (unsigned long long)ntile * (N / 64));
        atomicAdd(&p.counters[9], (unsigned long long)w_tfull);
        atomicAdd(&p.counters[11], (unsigned long long)(clock64() - t_start));
      }
    }
  }
  if (failed) atomicExch(p.status, GSKNN_ERR_TIMEOUT);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, (uint32_t)(2 * N));
}

// ------------------------------------------------------------------------------------------
// FP64 re-rank of the logged band
// ------------------------------------------------------------------------------------------
// What bounds it: latency and, in the batching form, issue. A query's band sits in NPART * S short
// logs, so a warp that walks them one after another waits for a count, then for a few entries,
// then for the next count. Here the counts are read at once and scanned, and the logs are read as one concatenated list.
//   1. entries at or under the partition bound + 2E go into a list in shared memory;
//   2. a bisection over the listed d' gives a bound on the approximate k-th close to it;
//   3. exact FP64 distances of the entries at or under that bound (about k of them), merged into
//      the sorted row; then of the entries above it, as far as they lie under the k-th of the
//      exact list + E.
// One warp per query (tc_rerank, tc_rerank_leaf), or one CTA per query when the queries are too
// few to fill the chip with warps (tc_rerank_cta).
// Measured against a warp that walked log after log with one lane per exact distance: 65,536 x
// 262,144, d = 64, k = 32: 751 -> 485 us; 32,768 x 262,144, d = 256, k = 64: 2,743 -> 1,246 us;
// 2,003 x 30,011: 119 -> 31 us; 16 x 4,096: 144 -> 15 us; 8 trees over 262,144 points: 9.4 -> 5.8 ms.
template <typename T>
struct RerankParams {
  int Q, k, S, logcap, d;
  const float4 *log;        // quads as the epilogue filtered them (log_mul)
  const uint32_t *logpos;   // packed position of each quad's first candidate
  const int *logcnt;
  const float *qn;
  const float *qmx;  // largest incoming distance of each query's heap row (tc_pack)
  int fold;             // the logged values are w (in the panels' scale), else v
  const float *fscale;  // as in TcParams
  int limit;  // double tables: a query with more candidates in its band goes to the next pass
  const unsigned *proot;  // partition roots of tc_knn ([query][S]; S counts NPART per split)
  const float *margin;
  const T *Xq, *Xq2, *Xc, *Xc2;
  long long nrows_q;
  const int *qidx;
  const uint32_t *cid;  // packed candidate position -> point id
  T *D;
  int *I;
  int ldD;
  int *fallback_list;
  int *fallback_count;
  unsigned long long *counters;  // optional: [5] entries scanned, [6] exact distances
  const int *dQ;      // optional: query count on the device (Q is then the stride)
  const int *rowmap;  // optional: heap row (and query position in qidx) of each query; -1: none
};

// d' of a logged value x: fma(log_mul, x, qn)
template <typename T>
__device__ __forceinline__ float log_mul(const RerankParams<T> &p) {
  const float fs = p.fscale ? *p.fscale : 1.0f;
  return p.fold ? -2.0f / (fs * fs) : 1.0f;
}

// (-2 <q,c> + |c|^2) + |q|^2, clamped at zero
__device__ __forceinline__ double exact_dist(double dot, double cc, double qq) {
  const double v = fma(-2.0, dot, cc) + qq;
  return v < 0.0 ? 0.0 : v;
}

// FP64 dot product of two float rows by four adjacent lanes (sub = lane & 3): lane `sub` sums the
// (exact) float x float products of every fourth group of four dimensions, then the four sums are
// added as a tree, so every candidate's value comes out of the same order of operations. Four lanes
// per row read 64 bytes of it side by side (a lane per row touches 32 lines with every load) and
// the FP64 chain is a quarter as long. All 32 lanes call it; every lane of the four gets the value.
__device__ __forceinline__ double exact_dot4(const float *q, const float *c, int d, int sub) {
  double acc = 0.0;
  const uintptr_t qc = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(c);
  if ((d & 3) == 0 && (qc & 15) == 0) {
    const float4 *q4 = reinterpret_cast<const float4 *>(q);
    const float4 *c4 = reinterpret_cast<const float4 *>(c);
#pragma unroll 4
    for (int i = sub; i < (d >> 2); i += 4) {
      const float4 a = __ldg(q4 + i), b = __ldg(c4 + i);
      acc = fma((double)a.x, (double)b.x, acc);
      acc = fma((double)a.y, (double)b.y, acc);
      acc = fma((double)a.z, (double)b.z, acc);
      acc = fma((double)a.w, (double)b.w, acc);
    }
  } else {
    for (int i = 4 * sub; i < d; i += 16)
      for (int pp = i; pp < min(i + 4, d); pp++) acc = fma((double)q[pp], (double)c[pp], acc);
  }
  return acc;
}
__device__ __forceinline__ double sum4(double acc) {
  acc += __shfl_xor_sync(FULL_MASK, acc, 1);
  acc += __shfl_xor_sync(FULL_MASK, acc, 2);
  return acc;
}

// The same dot product by one thread, in the same order (four sums over every fourth group of four
// dimensions, added as a tree): the brute-force passes. A query's distances are then the same bits
// whether its band fitted the logs or not. Summed in dimension order, as the brute force was when the
// re-rank did so too, about one neighbour in 10^8 came out another float.
__device__ __forceinline__ double dot_lane(const float *q, const float *c, int d) {
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  const uintptr_t qc = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(c);
  if ((d & 3) == 0 && (qc & 15) == 0) {
    const float4 *q4 = reinterpret_cast<const float4 *>(q);
    const float4 *c4 = reinterpret_cast<const float4 *>(c);
    for (int i = 0; i < (d >> 2); i += 4) {
#pragma unroll
      for (int s = 0; s < 4; s++) {
        if (i + s < (d >> 2)) {
          const float4 a = __ldg(q4 + i + s), b = __ldg(c4 + i + s);
          acc[s] = fma((double)a.x, (double)b.x, acc[s]);
          acc[s] = fma((double)a.y, (double)b.y, acc[s]);
          acc[s] = fma((double)a.z, (double)b.z, acc[s]);
          acc[s] = fma((double)a.w, (double)b.w, acc[s]);
        }
      }
    }
  } else {
    // sixteen loads of each row in flight: left to the compiler, the brute force's loop took 631 ms
    // on 16,384 x 60,000, d = 127, 196 so (rows of whole quads, d = 128: 472 ms a value at a time, 192)
    int p = 0;
    for (; p + 16 <= d; p += 16) {
      float a[16], b[16];
#pragma unroll
      for (int j = 0; j < 16; j++) {
        a[j] = __ldg(q + p + j);
        b[j] = __ldg(c + p + j);
      }
#pragma unroll
      for (int j = 0; j < 16; j++) acc[j >> 2] = fma((double)a[j], (double)b[j], acc[j >> 2]);
    }
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (p + j < d)
        acc[j >> 2] = fma((double)__ldg(q + p + j), (double)__ldg(c + p + j), acc[j >> 2]);
  }
  return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// FP64 dot product of two double rows by one thread, summed in dimension order: double tables, whose
// distances come out of the CUDA-core kernel's order of operations bit for bit.
__device__ __forceinline__ double dot_lane(const double *q, const double *c, int d) {
  double acc = 0.0;
  const uintptr_t qc = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(c);
  if ((d & 1) == 0 && (qc & 15) == 0) {
    const double2 *q2 = reinterpret_cast<const double2 *>(q);
    const double2 *c2 = reinterpret_cast<const double2 *>(c);
#pragma unroll 4
    for (int i = 0; i < (d >> 1); i++) {
      const double2 a = __ldg(q2 + i), b = __ldg(c2 + i);
      acc = fma(a.x, b.x, acc);
      acc = fma(a.y, b.y, acc);
    }
  } else {
#pragma unroll 4
    for (int pp = 0; pp < d; pp++) acc = fma(__ldg(q + pp), __ldg(c + pp), acc);
  }
  return acc;
}
__device__ __forceinline__ double exact_dist_lane(const float *q, const float *c, int d,
                                                  double cc, double qq) {
  return exact_dist(dot_lane(q, c, d), cc, qq);
}

// Order-preserving integer image of a double (-0 as 0, NaN last): the lists are sorted and merged
// by it, since a 64-bit integer comparison is two ALU instructions and an FP64 one goes through
// the narrow FP64 pipe.
typedef unsigned long long Ord;
constexpr Ord ORD_INF = 0xFFF0000000000000ull;  // image of +inf
__device__ __forceinline__ Ord to_ord(double x) {
  const Ord b = (Ord)__double_as_longlong(x), mag = b << 1;
  // (on the bits alone: tested as x != x in the branch of negative numbers, a NaN came out just below
  // 0 here, since the compiler may take either sign for it)
  if (mag > ORD_INF << 1 || mag == 0) return mag == 0 ? 0x8000000000000000ull : ~0ull;
  return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double from_ord(Ord o) {
  return __longlong_as_double((long long)((o >> 63) ? o & 0x7FFFFFFFFFFFFFFFull : ~o));
}

template <typename T, int E>
__device__ __forceinline__ void write_heap_row(T *D, int *I, int ldD, int q, int k,
                                               const Ord (&ld)[E], const uint32_t (&li)[E],
                                               int lane) {
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int t = e * 32 + lane;
    if (t < k) {
      D[(size_t)q * ldD + (k - 1 - t)] = (T)from_ord(ld[e]);
      I[(size_t)q * ldD + (k - 1 - t)] = (int)li[e];
    }
  }
}

// The heap row as it lies (reversed, so that the library's own descending rows come out
// ascending); the places past k hold (inf, NO_ID).
template <typename T, int E>
__device__ __forceinline__ void load_heap_row(const T *D, const int *I, int ldD, int q, int k,
                                              Ord (&ld)[E], uint32_t (&li)[E], int lane) {
#pragma unroll
  for (int e = 0; e < E; e++) {
    const int t = e * 32 + lane;
    if (t < k) {
      ld[e] = to_ord((double)D[(size_t)q * ldD + (k - 1 - t)]);
      li[e] = (uint32_t)I[(size_t)q * ldD + (k - 1 - t)];
    } else {
      ld[e] = ORD_INF;
      li[e] = NO_ID;
    }
  }
}

// Sorts the row ascending; a row that already is (an earlier call wrote it, or it is fresh) costs
// one comparison with each neighbour.
template <int E>
__device__ __forceinline__ void sort_heap_row(Ord (&ld)[E], uint32_t (&li)[E], int lane) {
  bool bad = false;
#pragma unroll
  for (int e = 0; e < E; e++) {
    Ord nd = __shfl_down_sync(FULL_MASK, ld[e], 1);
    uint32_t ni = __shfl_down_sync(FULL_MASK, li[e], 1);
    if (e + 1 < E) {
      const Ord fd = __shfl_sync(FULL_MASK, ld[e + 1 < E ? e + 1 : e], 0);
      const uint32_t fi = __shfl_sync(FULL_MASK, li[e + 1 < E ? e + 1 : e], 0);
      if (lane == 31) { nd = fd; ni = fi; }
    }
    if (lane < 31 || e + 1 < E) bad |= !(ld[e] < nd || (ld[e] == nd && li[e] <= ni));
  }
  if (__any_sync(FULL_MASK, bad)) warp_sort<Ord, E>(ld, li, lane);
}

// Sorts the first n of the warp's 32 keys ascending, the others being (inf, NO_ID): the bitonic
// network over the next power of two from eight on.
__device__ __forceinline__ void warp_sort_first(Ord &d, uint32_t &id, int n, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
    if (size > 8 && n <= size / 2) break;
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1)
      cx_shfl(d, id, stride, (lane & size) == 0, lane);
  }
}

// k-th smallest (0-based index k - 1) of the ascending list the warp holds
template <int E>
__device__ __forceinline__ Ord list_kth(const Ord (&ld)[E], int k) {
  Ord t = ld[0];
#pragma unroll
  for (int e = 0; e < E; e++)
    if (e == (k - 1) / 32) t = ld[e];
  return __shfl_sync(FULL_MASK, t, (k - 1) & 31);
}

// Largest value of the row (its k-th distance once it is full), as a float rounded up; -inf when
// all are NaN.
template <typename T>
__device__ __forceinline__ float row_max(const T *row, int k, int lane) {
  float mx = -Num<float>::inf();
  for (int j = lane; j < k; j += 32) mx = fmaxf(mx, up_f(row[j]));
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL_MASK, mx, o));
  return mx;
}

// Whether `id` (NO_ID: never) is one of the n ids in shared memory.
__device__ __forceinline__ bool id_in_row(uint32_t id, const uint32_t *ids, int n4) {
  const uint4 *v = reinterpret_cast<const uint4 *>(ids);
  bool a = false, b = false;
  for (int j = 0; j < n4; j++) {
    const uint4 x = v[j];
    a |= x.x == id || x.y == id;
    b |= x.z == id || x.w == id;
  }
  return (a || b) && id != NO_ID;
}

// A bound on the k-th smallest of the n >= k values list[i].x (as floats) with at most k + k/8 of
// them under it, or at most 1/4096 of their range above it; one warp.
__device__ __forceinline__ float list_bound(const uint2 *list, int n, int k, int lane) {
  float lo = Num<float>::inf(), hi = -Num<float>::inf();
  for (int i = lane; i < n; i += 32) {
    const float v = __uint_as_float(list[i].x);
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(FULL_MASK, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(FULL_MASK, hi, o));
  }
  for (int it = 0; it < 12; it++) {
    const float mid = lo + 0.5f * (hi - lo);
    int c = 0;
    for (int i = lane; i < n; i += 32) c += __uint_as_float(list[i].x) <= mid ? 1 : 0;
    c = __reduce_add_sync(FULL_MASK, c);
    if (c >= k) {
      hi = mid;
      if (c <= k + (k >> 3)) break;
    } else {
      lo = mid;
    }
  }
  return hi;
}

// Smallest and second smallest of the published partition roots over the warp's lanes.
__device__ __forceinline__ void two_smallest(unsigned &m1, unsigned &m2) {
  for (int o = 16; o; o >>= 1) {
    const unsigned a1 = __shfl_xor_sync(FULL_MASK, m1, o);
    const unsigned a2 = __shfl_xor_sync(FULL_MASK, m2, o);
    m2 = min(max(m1, a1), min(m2, a2));
    m1 = min(m1, a1);
  }
}

// the band: d' <= (bound on the approximate k-th) + 2E, and <= lim (a NaN bound admits nothing)
__device__ __forceinline__ float band_thr(float T, float E2, float lim) {
  const float t = __fadd_ru(T, E2);
  return lim < t ? lim : t;
}

// a row's largest distance + E bounds d' of any candidate that can still enter it
__device__ __forceinline__ float band_limit(float mx, float Eq) {
  return mx > -Num<float>::inf() && mx < 1e38f ? __fadd_ru(mx, Eq) : Num<float>::inf();
}

constexpr int RR_WARPS = 8;
// CTAs per SM the registers are held to: 64 registers up to 64 neighbours, 80 beyond (10,395 x 377,
// k = 114: 467 us with 128 registers, 308 with 80, 325 with 64)
template <int E>
constexpr int RR_OCC = E <= 2 ? 4 : 3;
template <int E>
constexpr int rr_cap() { return E == 1 ? 384 : 512; }  // listed entries per warp (k <= 32 E)

template <int E>
struct RerankSmem {
  uint2 list[rr_cap<E>()];     // (d', packed position)
  uint32_t stage[64];          // positions (batching form: ids) whose exact distances are next
  __align__(16) uint32_t ids[32 * E];  // batching form: the incoming row's ids
};

// One query by one warp. LEAF (the batching form): ids already in the row are not entered again,
// overflowed queries are listed by their panel rows, the incoming row stays unsorted until a
// candidate can enter it, and a row nothing entered is not written back.
template <typename Tab, int E, bool LEAF>
__device__ __forceinline__ void rerank_warp(const RerankParams<Tab> &p, int q, RerankSmem<E> &sm) {
  constexpr int CAP = rr_cap<E>();
  const int lane = threadIdx.x & 31;
  const int hr = p.rowmap ? p.rowmap[q] : q;  // heap row and query position
  // a padding row of a leaf panel, or a point outside the table (reported by tc_pack)
  if (hr < 0 || (LEAF && hr >= p.nrows_q)) return;
  const int k = p.k;
  Ord ld[E];
  uint32_t li[E];
  load_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
  bool ovf = false;
  unsigned m1 = 0xFFFFFFFFu, m2 = 0xFFFFFFFFu;
  for (int s = lane; s < p.S; s += 32) {
    ovf |= (p.logcnt[(size_t)s * p.Q + q] & (int)LOG_OVF) != 0;
    const unsigned u = p.proot[(size_t)q * p.S + s];
    m2 = min(m2, max(m1, u));
    m1 = min(m1, u);
  }
  const float E2 = p.margin[q], Eq = 0.5f * E2, qn = p.qn[q];
  // overflowed logs: the query goes to the next pass (a narrower format, or brute force); so does a
  // query whose bound left the floats' range or is NaN (the bound holds the maxima over all
  // candidates: one NaN coordinate makes every query's NaN, and nothing is logged)
  if (!(E2 < 1e38f)) ovf = true;
  if (__any_sync(FULL_MASK, ovf)) {
    if (lane == 0) p.fallback_list[atomicAdd(p.fallback_count, 1)] = LEAF ? q : hr;
    return;
  }
  // Any two heaps hold k candidates, so the second smallest final root bounds the approximate
  // k-th (all bits set: a heap that never filled). A candidate in the final top-k has d' <= the
  // approximate k-th + 2E, and d' <= (the k-th of any k exact distances) + E.
  if (LEAF) m2 = max(__shfl_sync(FULL_MASK, m1, 0), __shfl_sync(FULL_MASK, m1, 1));
  else two_smallest(m1, m2);
  float T = m2 == 0xFFFFFFFFu ? Num<float>::inf() : __uint_as_float(m2);
  const float mx = p.qmx[q];
  float lim = band_limit(mx, Eq);
  float thr = band_thr(T, E2, lim);
  Ord kth = to_ord((double)mx);  // of the exact list so far
  bool sorted = false;
  if (LEAF) {
#pragma unroll
    for (int e = 0; e < E; e++) sm.ids[e * 32 + lane] = li[e];
    __syncwarp();
  } else {
    sort_heap_row<E>(ld, li, lane);
    sorted = true;
  }
  const long long qrow = p.qidx[hr];
  if (qrow < 0 || qrow >= p.nrows_q) return;  // reported by tc_pack
  const Tab *qv = p.Xq + qrow * p.d;
  const double qq = (double)p.Xq2[qrow];
  const float qmul = log_mul(p);
  int n = 0;  // listed entries
  [[maybe_unused]] bool counted = false;

  // The logs, 32 at a time, as one concatenated list: lane s holds where log g + s starts. Entries
  // under the threshold fill the list; a full list is first cut down to what the bound from its
  // own entries admits, and if that is still most of it, or the logs are at their end, the exact
  // distances of the listed entries follow: those at or under the bound first (pass 0), then
  // those above it that the k-th of the exact list still admits.
  int g = -32, base = 0, total = 0, excl = 0;
  while (true) {
    bool done = false;
    while (n <= CAP - 128) {
      while (base >= total) {
        g += 32;
        if (g >= p.S) {
          done = true;
          break;
        }
        const int cnt = g + lane < p.S ? p.logcnt[(size_t)(g + lane) * p.Q + q] : 0;
        if (LEAF) {  // two logs: excl is where the second one starts
          excl = __shfl_sync(FULL_MASK, cnt, 0);
          total = excl + __shfl_sync(FULL_MASK, cnt, 1);
        } else {
          int incl = cnt;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL_MASK, incl, o);
            if (lane >= o) incl += v;
          }
          excl = incl - cnt;
          total = __shfl_sync(FULL_MASK, incl, 31);
        }
        base = 0;
        if (p.counters && lane == 0) atomicAdd(&p.counters[5], (unsigned long long)total);
      }
      if (done) break;
      const int e = base + lane;
      int s = 0, off;  // the last log that starts at or before e, and e's place in it
      if (LEAF) {
        s = e >= excl ? 1 : 0;
        off = e - (s ? excl : 0);
      } else {
#pragma unroll
        for (int st = 16; st; st >>= 1) {
          const int v = __shfl_sync(FULL_MASK, excl, s + st);
          if (v <= e) s += st;
        }
        off = e - __shfl_sync(FULL_MASK, excl, s);
      }
      float dv[4];
      uint32_t pos = 0u;
      {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (e < total) {
          const size_t at = ((size_t)(g + s) * p.Q + q) * p.logcap + off;
          v = p.log[at];
          pos = p.logpos[at];
        }
        dv[0] = fmaf(qmul, v.x, qn);
        dv[1] = fmaf(qmul, v.y, qn);
        dv[2] = fmaf(qmul, v.z, qn);
        dv[3] = fmaf(qmul, v.w, qn);
      }
      base += 32;
      if (!__any_sync(FULL_MASK,
                      e < total && fminf(fmin3(dv[0], dv[1], dv[2]), dv[3]) <= thr))
        continue;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const bool take = e < total && dv[u] <= thr;
        const unsigned m = __ballot_sync(FULL_MASK, take);
        if (take)
          sm.list[n + __popc(m & ((1u << lane) - 1u))] =
              make_uint2(__float_as_uint(dv[u]), pos + u);
        n += __popc(m);
      }
    }
    __syncwarp();
    // (a full row of the batching form bounds its candidates itself: most of those it admits are in
    // it already, so that the rest is one short batch)
    const bool bound = n > 32 && !(LEAF && lim < Num<float>::inf());
    if (bound && n >= k) T = fminf(T, fmaxf(list_bound(sm.list, n, k, lane), 0.0f));
    thr = band_thr(T, E2, lim);
    const float split = bound ? T : Num<float>::inf();  // one batch takes a short list whole
    if (!done) {
      int w = 0;
      for (int b0 = 0; b0 < n; b0 += 32) {
        const int e = b0 + lane;
        const uint2 ent = e < n ? sm.list[e] : make_uint2(0u, 0u);
        const bool keep = e < n && __uint_as_float(ent.x) <= thr;
        const unsigned m = __ballot_sync(FULL_MASK, keep);
        if (keep) sm.list[w + __popc(m & ((1u << lane) - 1u))] = ent;
        w += __popc(m);
        __syncwarp();
      }
      n = w;
      if (n <= CAP / 2) continue;
      // A band that fills the list: a double query whose band is a large part of the candidates
      // (points closer than the rounding of their own distances) leaves before its first exact
      // distance, not with its whole band's (band_limit_of). Counted are the candidates within 2E
      // of the nearest one, which are in the band whatever the k-th turns out to be.
      if constexpr (sizeof(Tab) == 8) {
        if (!counted) {
          counted = true;
          float lo = Num<float>::inf();
          int c = 0;
          for (int sweep = 0; sweep < 2; sweep++) {
            const float t = __fadd_rd(fmaxf(lo, 0.0f), E2);
            for (int s = 0; s < p.S; s++) {
              const int cnt = p.logcnt[(size_t)s * p.Q + q];
              const float4 *const lg = p.log + ((size_t)s * p.Q + q) * p.logcap;
              for (int e = lane; e < cnt; e += 32) {
                const float4 v = lg[e];
                const float d0 = fmaf(qmul, v.x, qn), d1 = fmaf(qmul, v.y, qn),
                            d2 = fmaf(qmul, v.z, qn), d3 = fmaf(qmul, v.w, qn);
                if (sweep == 0) lo = fminf(lo, fminf(fmin3(d0, d1, d2), d3));
                else c += (d0 <= t) + (d1 <= t) + (d2 <= t) + (d3 <= t);
              }
            }
            if (sweep == 0)
              for (int o = 16; o; o >>= 1) lo = fminf(lo, __shfl_xor_sync(FULL_MASK, lo, o));
          }
          if (__reduce_add_sync(FULL_MASK, c) > p.limit) {
            if (lane == 0) p.fallback_list[atomicAdd(p.fallback_count, 1)] = hr;
            return;
          }
        }
      }
    }
    int nb = 0;  // staged candidates
    const int nblk = (n + 31) / 32;
    for (int i = 0; i < (bound ? 2 * nblk : nblk); i++) {
      const bool pass1 = i >= nblk;
      const int e = (pass1 ? i - nblk : i) * 32 + lane;
      uint32_t id = NO_ID;
      if (e < n) {
        const uint2 ent = sm.list[e];
        const float dv = __uint_as_float(ent.x);
        if (dv <= thr && (dv > split) == pass1) id = LEAF ? p.cid[ent.y] : ent.y;
      }
      // an id already in the incoming row costs no row gather
      if (LEAF && id_in_row(id, sm.ids, 8 * E)) id = NO_ID;
      const unsigned m = __ballot_sync(FULL_MASK, id != NO_ID);
      if (id != NO_ID) sm.stage[nb + __popc(m & ((1u << lane) - 1u))] = id;
      nb += __popc(m);
      __syncwarp();
      const bool end = i == nblk - 1 || i == 2 * nblk - 1;
      while (nb >= 32 || (end && nb > 0)) {
        // exact distances of these candidates, merged into the list: lane i takes candidate i's
        // norm, four lanes its dot product
        const int cnt = nb < 32 ? nb : 32;
        id = lane < cnt ? (LEAF ? sm.stage[lane] : p.cid[sm.stage[lane]]) : NO_ID;
        const uint32_t rest = sm.stage[32 + lane];
        __syncwarp();
        sm.stage[lane] = rest;
        nb -= cnt;
        __syncwarp();
        const double cc = id != NO_ID ? (double)p.Xc2[id] : 0.0;
        double dot = 0.0;
        if constexpr (sizeof(Tab) == 8) {
          if (id != NO_ID) dot = dot_lane(qv, p.Xc + (long long)id * p.d, p.d);
        } else for (int r = 0; r < cnt; r += 8) {
          const uint32_t cid = __shfl_sync(FULL_MASK, id, r + (lane >> 2));
          double part = 0.0;
          if (cid != NO_ID)
            part = exact_dot4(qv, p.Xc + (long long)cid * p.d, p.d, lane & 3);
          part = __shfl_sync(FULL_MASK, sum4(part), (lane & 7) * 4);
          if ((lane >> 3) == (r >> 3)) dot = part;
        }
        const Ord dist = id != NO_ID ? to_ord(exact_dist(dot, cc, qq)) : ORD_INF;
        if (p.counters && lane == 0) atomicAdd(&p.counters[6], (unsigned long long)cnt);
        if (LEAF) {
          // nothing in this batch can enter (ties are settled by the merge itself)
          if (!__any_sync(FULL_MASK, id != NO_ID && dist <= kth)) continue;
          if (!sorted) {
            sort_heap_row<E>(ld, li, lane);
            sorted = true;
          }
        }
        Ord bd = dist;
        uint32_t bi = id;
        warp_sort_first(bd, bi, cnt, lane);
        warp_merge_32<Ord, E>(ld, li, bd, bi, lane);
        kth = list_kth<E>(ld, k);
        const double kd = from_ord(kth);
        if (kd < 1e38) {
          lim = fminf(lim, __fadd_ru(__double2float_ru(kd), Eq));
          if (lim < thr) thr = lim;
        }
      }
    }
    if (done) break;
    n = 0;
    __syncwarp();
  }
  if (sorted) write_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
}

template <typename Tab, int E>
__global__ void __launch_bounds__(32 * RR_WARPS, RR_OCC<E>) tc_rerank(RerankParams<Tab> p) {
  __shared__ RerankSmem<E> sm[RR_WARPS];
  const int q = blockIdx.x * RR_WARPS + (threadIdx.x >> 5);
  if (q >= (p.dQ ? *p.dQ : p.Q)) return;
  rerank_warp<Tab, E, false>(p, q, sm[threadIdx.x >> 5]);
}

template <int E>
__global__ void __launch_bounds__(32 * RR_WARPS, RR_OCC<E>) tc_rerank_leaf(RerankParams<float> p) {
  __shared__ RerankSmem<E> sm[RR_WARPS];
  const int q = blockIdx.x * RR_WARPS + (threadIdx.x >> 5);
  if (q >= p.Q) return;
  rerank_warp<float, E, true>(p, q, sm[threadIdx.x >> 5]);
}

// One query by one CTA: all warps read the logs into one list and share the exact distances; warp
// 0 merges.
constexpr int RC_CAP = 1024;  // listed entries per CTA
constexpr int RC_LOGS = 512;  // logs (NPART * S) the prefix array holds

template <typename Tab, int E>
__global__ void __launch_bounds__(32 * RR_WARPS, RR_OCC<E>) tc_rerank_cta(RerankParams<Tab> p) {
  __shared__ uint2 list[RC_CAP];
  __shared__ Ord xd[RC_CAP];
  __shared__ uint32_t xi[RC_CAP];
  __shared__ Ord hold_d[32 * E];  // the list between the rounds of a wide band
  __shared__ uint32_t hold_i[32 * E];
  __shared__ int pre[RC_LOGS + 1];
  __shared__ float s_T, s_thr;
  __shared__ int s_n, s_state;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int q = blockIdx.x;
  if (q >= (p.dQ ? *p.dQ : p.Q)) return;
  const int hr = p.rowmap ? p.rowmap[q] : q;
  if (hr < 0) return;
  const int k = p.k;
  const float E2 = p.margin[q], Eq = 0.5f * E2, qn = p.qn[q];
  if (warp == 0) {
    // prefix sums of the counts, the overflow flag and the partition bound
    bool ovf = false;
    unsigned m1 = 0xFFFFFFFFu, m2 = 0xFFFFFFFFu;
    int carry = 0;
    for (int g = 0; g < p.S; g += 32) {
      int c = 0;
      if (g + lane < p.S) {
        c = p.logcnt[(size_t)(g + lane) * p.Q + q];
        ovf |= (c & (int)LOG_OVF) != 0;
        const unsigned u = p.proot[(size_t)q * p.S + g + lane];
        m2 = min(m2, max(m1, u));
        m1 = min(m1, u);
      }
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL_MASK, incl, o);
        if (lane >= o) incl += v;
      }
      if (g + lane < p.S) pre[g + lane + 1] = carry + incl;
      carry += __shfl_sync(FULL_MASK, incl, 31);
    }
    ovf = __any_sync(FULL_MASK, ovf) || !(E2 < 1e38f);
    two_smallest(m1, m2);
    const float T = m2 == 0xFFFFFFFFu ? Num<float>::inf() : __uint_as_float(m2);
    const float lim = band_limit(row_max(p.D + (size_t)hr * p.ldD, k, lane), Eq);
    if (lane == 0) {
      pre[0] = 0;
      s_T = T;
      s_thr = band_thr(T, E2, lim);
      s_n = 0;
      s_state = ovf ? 1 : 0;
      if (ovf) p.fallback_list[atomicAdd(p.fallback_count, 1)] = hr;
      if (p.counters) atomicAdd(&p.counters[5], (unsigned long long)carry);
    }
  }
  __syncthreads();
  if (s_state) return;
  const long long qrow = p.qidx[hr];
  if (qrow < 0 || qrow >= p.nrows_q) return;  // reported by tc_pack
  const Tab *qv = p.Xq + qrow * p.d;
  const double qq = (double)p.Xq2[qrow];
  const int total = pre[p.S];
  float thr = s_thr;
  const float qmul = log_mul(p);
  // lists the entries under thr of the quads e0 .. e1; s_n counts them all
  auto gather = [&](int e0, int e1) {
    for (int e = e0 + tid; e < e1; e += 32 * RR_WARPS) {
      int a = 0, b = p.S;  // the last log that starts at or before e
      while (b - a > 1) {
        const int m = (a + b) >> 1;
        if (pre[m] <= e) a = m;
        else b = m;
      }
      const size_t at = ((size_t)a * p.Q + q) * p.logcap + (e - pre[a]);
      const float4 v4 = p.log[at];
      const uint32_t pos = p.logpos[at];
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const float dv = fmaf(qmul, v[u], qn);
        if (dv <= thr) {
          const int to = atomicAdd(&s_n, 1);
          if (to < RC_CAP) list[to] = make_uint2(__float_as_uint(dv), pos + u);
        }
      }
    }
    __syncthreads();
  };
  gather(0, total);
  int n = s_n;
  // The partition bound is loose where long lists meet many short splits: entries that fill the list
  // bound the k-th far better, and what is left under their bound mostly fits (2 x 13,650, d = 141,
  // k = 100 321 us without this, 186).
  for (int pass = 0; n > RC_CAP && pass < 3; pass++) {
    __syncthreads();  // every thread has read the count that warp 0 resets
    if (warp == 0) {
      const float T = fminf(s_T, fmaxf(list_bound(list, RC_CAP, k, lane), 0.0f));
      if (lane == 0) {
        s_T = T;
        s_thr = band_thr(T, E2, thr);
        s_n = 0;
      }
    }
    __syncthreads();
    if (!(s_thr < thr)) {
      if (tid == 0) s_n = n;
      __syncthreads();
      break;
    }
    thr = s_thr;
    gather(0, total);
    n = s_n;
  }
  // A band that does not fit the list is taken a quarter of the list's quads at a time (by one warp
  // alone, as a list it fills again and again, 0.25 us an exact distance: 500 double queries x 50,021,
  // d = 32, k = 50, clusters of 3,100 965 us, 646 so); of a double query, only if it is a small
  // part of the candidates (band_limit_of).
  const bool whole = n <= RC_CAP;
  if (!whole && sizeof(Tab) == 8 && n > p.limit) {
    if (tid == 0) p.fallback_list[atomicAdd(p.fallback_count, 1)] = hr;
    return;
  }
  if (whole && n > 32 && n >= k) {
    if (warp == 0) {
      const float T = fminf(s_T, fmaxf(list_bound(list, n, k, lane), 0.0f));
      if (lane == 0) s_thr = band_thr(T, E2, thr);
    }
    __syncthreads();
    thr = s_thr;
  }
  constexpr int LPC = sizeof(Tab) == 8 ? 1 : 4;  // lanes per candidate
  // exact distances of the listed entries under thr, by all warps
  auto exact = [&]() {
    for (int base = warp * (32 / LPC); base < n; base += 32 / LPC * RR_WARPS) {
      const int i = base + lane / LPC;
      uint32_t id = NO_ID;
      if (i < n && __uint_as_float(list[i].x) <= thr) id = p.cid[list[i].y];
      double dot = 0.0;
      if constexpr (LPC == 1) {
        if (id != NO_ID) dot = dot_lane(qv, p.Xc + (long long)id * p.d, p.d);
      } else {
        if (id != NO_ID) dot = exact_dot4(qv, p.Xc + (long long)id * p.d, p.d, lane & 3);
        dot = sum4(dot);
      }
      if (i < n && lane % LPC == 0) {
        xd[i] = id != NO_ID ? to_ord(exact_dist(dot, (double)p.Xc2[id], qq)) : ORD_INF;
        xi[i] = id;
        if (p.counters && id != NO_ID) atomicAdd(&p.counters[6], 1ull);
      }
    }
    __syncthreads();
  };
  Ord ld[E];
  uint32_t li[E];
  // merges them into the list, by warp 0
  auto merge = [&](Ord kth) {
    for (int base = 0; base < n; base += 32) {
      const int i = base + lane;
      Ord b1[1] = {i < n ? xd[i] : ORD_INF};
      uint32_t i1[1] = {i < n ? xi[i] : NO_ID};
      if (!__any_sync(FULL_MASK, i1[0] != NO_ID && b1[0] <= kth)) continue;
      warp_sort<Ord, 1>(b1, i1, lane);
      warp_merge_32<Ord, E>(ld, li, b1[0], i1[0], lane);
      kth = list_kth<E>(ld, k);
    }
    return kth;
  };
  if (whole) {
    exact();
    if (warp != 0) return;
    load_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
    sort_heap_row<E>(ld, li, lane);
    merge(list_kth<E>(ld, k));
    write_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
    return;
  }
  // The list waits in shared memory between the rounds (kept in registers across them, the exact
  // distances of every other call were a third slower).
  constexpr int STEP = RC_CAP / 4;
  if (warp == 0) {
    load_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
    sort_heap_row<E>(ld, li, lane);
#pragma unroll
    for (int e = 0; e < E; e++) {
      hold_d[e * 32 + lane] = ld[e];
      hold_i[e * 32 + lane] = li[e];
    }
  }
  for (int e0 = 0; e0 < total; e0 += STEP) {
    __syncthreads();  // warp 0 is done with the last round
    if (tid == 0) s_n = 0;
    thr = s_thr;
    __syncthreads();
    gather(e0, min(total, e0 + STEP));
    n = s_n;
    if (n == 0) continue;
    exact();
    if (warp == 0) {
#pragma unroll
      for (int e = 0; e < E; e++) {
        ld[e] = hold_d[e * 32 + lane];
        li[e] = hold_i[e * 32 + lane];
      }
      const double kd = from_ord(merge(list_kth<E>(ld, k)));
#pragma unroll
      for (int e = 0; e < E; e++) {
        hold_d[e * 32 + lane] = ld[e];
        hold_i[e * 32 + lane] = li[e];
      }
      if (lane == 0 && kd < 1e38) s_thr = fminf(s_thr, __fadd_ru(__double2float_ru(kd), Eq));
    }
  }
  if (warp == 0) {
#pragma unroll
    for (int e = 0; e < E; e++) {
      ld[e] = hold_d[e * 32 + lane];
      li[e] = hold_i[e * 32 + lane];
    }
    write_heap_row<Tab, E>(p.D, p.I, p.ldD, hr, k, ld, li, lane);
  }
}

// ------------------------------------------------------------------------------------------
// exact brute force for queries whose log overflowed (rare; one CTA per query)
// ------------------------------------------------------------------------------------------
struct FallbackParams {
  int k, d, nc;
  const float *Xq, *Xq2, *Xc, *Xc2;
  const int *qidx, *cidx;
  long long nrows_q, nrows_c;
  float *D;
  int *I;
  int ldD;
  const int *list;
  const int *count;
  const int *status;  // the call's status word, copied to the host-visible mirror (may be null):
  int *mirror;        // this is the call's last kernel
};

template <int E>
__global__ void __launch_bounds__(256) tc_fallback(FallbackParams p) {
  if (p.mirror && blockIdx.x == 0 && threadIdx.x == 0) *p.mirror = *p.status;
  __shared__ Ord sd[8][32 * E];
  __shared__ uint32_t si[8][32 * E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = *p.count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int q = p.list[w];
    const long long qrow = p.qidx[q];
    if (qrow < 0 || qrow >= p.nrows_q) continue;  // reported by tc_pack
    const float *qv = p.Xq + qrow * p.d;
    const double qq = (double)p.Xq2[qrow];
    Ord ld[E];
    uint32_t li[E];
#pragma unroll
    for (int e = 0; e < E; e++) { ld[e] = ORD_INF; li[e] = NO_ID; }
    Ord kth = ORD_INF;
    // each warp scans a strided share of the candidates, one candidate per lane at a time
    for (int base = warp * 32; base < p.nc; base += 256) {
      const int c = base + lane;
      double dist = Num<double>::inf();
      uint32_t id = NO_ID;
      if (c < p.nc) {
        const long long row = p.cidx[c];
        if (row >= 0 && row < p.nrows_c) {
          dist = exact_dist_lane(qv, p.Xc + row * p.d, p.d, (double)p.Xc2[row], qq);
          id = (uint32_t)row;
        }
      }
      Ord b1[1] = {to_ord(dist)};
      if (__any_sync(FULL_MASK, b1[0] <= kth)) {
        uint32_t i1[1] = {id};
        warp_sort<Ord, 1>(b1, i1, lane);
        warp_merge_32<Ord, E>(ld, li, b1[0], i1[0], lane);
        kth = list_kth<E>(ld, p.k);
      }
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
      sd[warp][e * 32 + lane] = ld[e];
      si[warp][e * 32 + lane] = li[e];
    }
    __syncthreads();
    if (warp == 0) {
      Ord md[E];
      uint32_t mi[E];
      load_heap_row<float, E>(p.D, p.I, p.ldD, q, p.k, md, mi, lane);
      sort_heap_row<E>(md, mi, lane);
      for (int w2 = 0; w2 < 8; w2++) {
        Ord bd[E];
        uint32_t bi[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
          bd[e] = sd[w2][e * 32 + lane];
          bi[e] = si[w2][e * 32 + lane];
        }
        warp_merge_lists<Ord, E>(md, mi, bd, bi, lane);
      }
      write_heap_row<float, E>(p.D, p.I, p.ldD, q, p.k, md, mi, lane);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------
// batching form: exact brute force of overflowed queries over their own leaf
// ------------------------------------------------------------------------------------------
struct LeafFallbackParams {
  int k, d, N;                 // N: candidate tile width of the panel
  const float *X, *X2;         // the point table
  const int *rowmap;           // panel row -> point (heap row)
  const uint32_t *ids;         // panel row -> point id (NO_ID: padding)
  const int2 *rtab;            // panel query tile -> (first, end) candidate tile of its leaf
  float *D;
  int *I;
  int ldD;
  const int *list;             // panel rows
  const int *count;
};

// One warp per listed query: the exact FP64 distances to every point of its leaf, merged with
// the incoming heap row (ids already there are not entered twice).
template <int E>
__global__ void __launch_bounds__(256) tc_fallback_leaf(LeafFallbackParams p) {
  const int lane = threadIdx.x & 31;
  const int n = *p.count;
  for (int w = blockIdx.x * 8 + (threadIdx.x >> 5); w < n; w += gridDim.x * 8) {
    const int q = p.list[w];
    const int hr = p.rowmap[q];
    const int2 r = p.rtab[q / TC_M];
    const float *qv = p.X + (long long)hr * p.d;
    const double qq = (double)p.X2[hr];
    Ord ld[E];
    uint32_t li[E];
    load_heap_row<float, E>(p.D, p.I, p.ldD, hr, p.k, ld, li, lane);
    sort_heap_row<E>(ld, li, lane);
    __shared__ __align__(16) uint32_t ids[8][32 * E];  // the incoming row's ids
    uint32_t *const li0 = ids[threadIdx.x >> 5];
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; e++) li0[e * 32 + lane] = li[e];
    __syncwarp();
    for (int base = r.x * p.N; base < r.y * p.N; base += 32) {  // warp-uniform trip count
      const int c = base + lane;
      uint32_t id = NO_ID;
      double dist = Num<double>::inf();
      if (c < r.y * p.N) {
        id = p.ids[c];
        if (id != NO_ID)
          dist = exact_dist_lane(qv, p.X + (long long)id * p.d, p.d, (double)p.X2[id], qq);
      }
      if (id_in_row(id, li0, 8 * E)) {
        dist = Num<double>::inf();
        id = NO_ID;
      }
      Ord b1[1] = {to_ord(dist)};
      uint32_t i1[1] = {id};
      warp_sort<Ord, 1>(b1, i1, lane);
      warp_merge_32<Ord, E>(ld, li, b1[0], i1[0], lane);
    }
    write_heap_row<float, E>(p.D, p.I, p.ldD, hr, p.k, ld, li, lane);
  }
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// Row-major [rows][d_pad] panel of elem-byte elements; box = 128 bytes x box_rows rows, 128B
// swizzle (the K-major layout tcgen05 descriptors expect).
static cudaError_t make_panel_map(CUtensorMap *m, void *base, int elem, int d_pad, int rows,
                                  int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t gdim[2] = {(cuuint64_t)d_pad, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)d_pad * elem};
  cuuint32_t box[2] = {(cuuint32_t)(CHUNK_BYTES / elem), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16,
                  2, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Norm panel [rows][32 bytes] (write_norm_row), box of box_rows rows, 32-byte swizzle.
static cudaError_t make_norm_map(CUtensorMap *m, void *base, int elem, int rows, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t gdim[2] = {(cuuint64_t)(NORM_ROW / elem), (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)NORM_ROW};
  cuuint32_t box[2] = {(cuuint32_t)(NORM_ROW / elem), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16,
                  2, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Launches tc_knn in the plan's format, with the norm column when `npanel` (the candidates' norm
// panel) is given and its areas fit; sets the matching error-bound coefficients in tp.
template <typename Grid>
static cudaError_t launch_tc_knn(const TcPlan &P, void *npanel, int npanel_rows, Grid grid,
                                 const CUtensorMap &mA, const CUtensorMap &mAlo,
                                 const CUtensorMap &mB, const CUtensorMap &mBlo, TcParams &tp,
                                 cudaStream_t st) {
  const bool fold = npanel && P.smem_fold;
  CUtensorMap mBn = mB;
  if (fold) {
    const cudaError_t e = make_norm_map(&mBn, npanel, P.elem, npanel_rows, P.N);
    if (e != cudaSuccess) return e;
  }
  tp.fold = fold ? 1 : 0;
  tp.kC = P.kB + (fold ? P.kC_fold : 0.0f);
  tp.kS = P.kS;
  const unsigned smem = fold ? P.smem_fold : P.smem;
  cudaError_t e = cudaSuccess;
  auto go = [&](auto kern) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) kern<<<grid, NTHREADS, smem, st>>>(mA, mAlo, mB, mBlo, mBn, tp);
  };
  if (P.fmt == 0)
    fold ? go(tc_knn<0, true, true>) : P.ringed ? go(tc_knn<0, false, true>)
                                                : go(tc_knn<0, false, false>);
  else if (P.fmt != 2)
    fold ? go(tc_knn<1, true, true>) : P.ringed ? go(tc_knn<1, false, true>)
                                                : go(tc_knn<1, false, false>);
  else
    fold ? go(tc_knn<2, true, true>) : P.ringed ? go(tc_knn<2, false, true>)
                                                : go(tc_knn<2, false, false>);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e;
}

}  // namespace tc

static size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

int tc_format_of_mode(int mode) {
  return mode == GSKNN_TC_BF16 ? 1 : mode == GSKNN_TC_BF16X3 ? 2 : mode == GSKNN_TC_FP16 ? 3 : 0;
}

// Prepared-candidate area: shift, FP16 scale, stats, panel(s), norms, ids.
struct CandLayout {
  size_t o_mu, o_fscale, o_cpart, o_stats, o_pb, o_pb_lo, o_pn, o_cn, o_cid, bytes;
  int fmt, elem, d_pad, r_pad;
};

static CandLayout cand_layout(int nc, int d, int mode) {
  using namespace tc;
  CandLayout L{};
  L.fmt = tc_format_of_mode(mode);
  L.elem = L.fmt == 0 ? 4 : 2;
  const int celems = CHUNK_BYTES / L.elem;
  L.d_pad = ((d + celems - 1) / celems) * celems;
  L.r_pad = ((nc + 255) / 256) * 256;  // whole tiles of 256 and of 128 candidates
  size_t off = 0;
  auto take = [&](size_t b) { size_t o = off; off = al256(off + b); return o; };
  L.o_mu = take((size_t)d * 4);
  L.o_fscale = take(8);
  L.o_cpart = take((size_t)CENTER_PARTS * d * 8 + CENTER_SLICES * 4);
  L.o_stats = take(2 * STATS_WORDS * 4);
  L.o_pb = take((size_t)L.r_pad * L.d_pad * L.elem);
  L.o_pb_lo = L.fmt == 2 ? take((size_t)L.r_pad * L.d_pad * L.elem) : 0;
  L.o_pn = take((size_t)L.r_pad * NORM_ROW);
  L.o_cn = take((size_t)L.r_pad * 4);
  L.o_cid = take((size_t)L.r_pad * 4);
  L.bytes = off;
  return L;
}

static int tc_mode_of_format(int fmt) {
  return fmt == 1   ? GSKNN_TC_BF16
         : fmt == 2 ? GSKNN_TC_BF16X3
         : fmt == 3 ? GSKNN_TC_FP16
                    : GSKNN_TC_TF32;
}

size_t tc_cand_bytes(int nc, int d, int mode) { return cand_layout(nc, d, mode).bytes; }

// Lays out candidates in `mem` (cand_layout) and enqueues their shift.
template <typename T>
static cudaError_t cand_begin(TcCand *C, void *mem, int nc, int d, int mode, const T *Xc,
                              const T *Xc2, long long nrows_c, const int *cidx, int *clear,
                              cudaStream_t st) {
  using namespace tc;
  const CandLayout L = cand_layout(nc, d, mode);
  char *base = static_cast<char *>(mem);
  C->fmt = L.fmt; C->elem = L.elem; C->d = d; C->d_pad = L.d_pad; C->nc = nc; C->r_pad = L.r_pad;
  C->mu = reinterpret_cast<float *>(base + L.o_mu);
  C->part = reinterpret_cast<double *>(base + L.o_cpart);
  C->part_n = reinterpret_cast<int *>(base + L.o_cpart + (size_t)CENTER_PARTS * d * 8);
  C->stats = reinterpret_cast<unsigned *>(base + L.o_stats);
  C->estats = C->stats + STATS_WORDS;
  C->fscale = reinterpret_cast<float *>(base + L.o_fscale);
  C->pb = base + L.o_pb;
  C->pb_lo = L.fmt == 2 ? base + L.o_pb_lo : nullptr;
  C->pn = base + L.o_pn;
  C->cn = reinterpret_cast<float *>(base + L.o_cn);
  C->cid = reinterpret_cast<uint32_t *>(base + L.o_cid);
  C->Xc = Xc; C->Xc2 = Xc2; C->nrows_c = nrows_c; C->cidx = cidx;
  C->efmt = -1; C->epb = nullptr; C->epb_lo = nullptr; C->epn = nullptr;
  tc_center<T><<<dim3((d + 31) / 32, CENTER_SLICES), 32 * CENTER_WARPS, 0, st>>>(
      Xc, d, nrows_c, cidx, nc, std::min(nc, CENTER_ROWS), C->part, C->part_n, C->stats,
      2 * STATS_WORDS, clear);
  return cudaGetLastError();
}

// The candidates' side of a packing launch, in their main format.
template <typename T>
static tc::PackSide<T> cand_side(const TcCand &C) {
  tc::PackSide<T> s{};
  s.X = static_cast<const T *>(C.Xc);
  s.X2 = static_cast<const T *>(C.Xc2);
  s.nrows = C.nrows_c;
  s.idx = C.cidx;
  s.count = C.nc;
  s.rows_pad = C.r_pad;
  s.panel = C.pb;
  s.panel_lo = C.pb_lo;
  s.npanel = C.pn;
  s.enorm = C.cn;
  s.ids = C.cid;
  s.stats = C.stats;
  return s;
}

// Packs one side or both; with `sums` the shift comes from the partial sums of tc_center.
template <typename T>
static cudaError_t launch_tc_pack(const tc::PackSide<T> &a, const tc::PackSide<T> &b,
                                  const TcCand &C, int fmt, int d_pad, bool sums, float kA,
                                  float kB, float kS, int *status, cudaStream_t st) {
  tc::PackArgs<T> g{};
  g.fmt = fmt;
  g.d = C.d;
  g.d_pad = d_pad;
  g.a = a;
  g.b = b;
  g.part = sums ? C.part : nullptr;
  g.part_n = C.part_n;
  g.mu = C.mu;
  g.fscale = C.fscale;
  g.kA = kA;
  g.kB = kB;
  g.kS = kS;
  g.status = status;
  tc::tc_pack<T><<<tc::tc_pack_grid((long long)a.rows_pad + b.rows_pad), 256,
                   (size_t)C.d * sizeof(double), st>>>(g);
  return cudaGetLastError();
}

cudaError_t tc_cand_prepare(TcCand *C, void *mem, int nc, int d, int mode, const float *Xc,
                            const float *Xc2, long long nrows_c, const int *cidx, int *status,
                            cudaStream_t st) {
  const cudaError_t e =
      cand_begin<float>(C, mem, nc, d, mode, Xc, Xc2, nrows_c, cidx, nullptr, st);
  if (e != cudaSuccess) return e;
  return launch_tc_pack<float>(cand_side<float>(*C), tc::PackSide<float>{}, *C, C->fmt, C->d_pad,
                               true, 0.0f, 0.0f, 0.0f, status, st);
}

// Quads per log: `want`, or in a tight plan those that fit the 8 * want bytes of as many single
// candidates, but not fewer than twice the room that two chunks want.
static int log_entries(int want, bool tight) {
  return tight ? std::max((int)(want * 8 / tc::LOG_ENTRY), 2 * tc::LOG_ROOM) : want;
}

static TcPlan tc_plan_base(int nq, int nc, int d, int k, int mode, int sms, bool with_cand,
                          int max_splits, bool tight = false) {
  using namespace tc;
  TcPlan P{};
  P.ok = false;
  P.sms = sms;
  P.max_splits = max_splits;
  P.tight = tight;
  P.fmt = tc_format_of_mode(mode);
  const int elem = P.fmt == 0 ? 4 : 2;
  const int celems = CHUNK_BYTES / elem;
  P.elem = elem;
  P.d_pad = ((d + celems - 1) / celems) * celems;
  P.nkc = P.d_pad / celems;
  P.a_terms = P.fmt == 2 ? 2 : 1;
  P.kp = 32;
  while (P.kp < k) P.kp <<= 1;
  if (k > 256) return P;
  // Candidate tile width and pipeline depth that fit in shared memory, and whether the norm column
  // fits beside them: in split BF16 and FP16, and in BF16 from two K chunks (measured in tc_knn:
  // split BF16 at d = 64 -4%, BF16 at d = 256 -1.6%, but BF16 at d = 64 +5%; split BF16 at d = 64
  // with five stages in place of the norm column 6,320 us against 5,931). Three stages of the
  // pipeline are worth less than the norm column's areas.
  const uint32_t smem_max = 227 * 1024;
  const int lists = NPART * list_slots(tc_heap_k(k));
  bool fold = P.fmt >= 2 || (P.fmt == 1 && P.nkc >= 2);
  if (const char *v = getenv("GSKNN_TC_FOLD"))
    if (atoi(v) == 0) fold = false;
  // The limit of the format: two chunks of every term in flight, at the narrow tile.
  const int least = 2 * P.a_terms;
  if (tc_smem_layout(P.nkc, P.a_terms, 128, least, lists, false, false).total > smem_max) return P;
  int best_N = 0, best_NST = 0;
  uint32_t smem_fold = 0;
  const int Ns[2] = {256, 128};
  for (int ni = 0; ni < 2 && !best_N; ni++) {
    const int N = Ns[ni];
    if (P.fmt == 0 && N == 256 && P.nkc > 4) continue;  // keep the TF32 A tile room
    for (int NST = 6; NST >= 2 && !best_N; NST--) {
      const uint32_t with = tc_smem_layout(P.nkc, P.a_terms, N, NST, lists, true, true).total;
      if (fold && with <= smem_max && NST >= 3) {
        best_N = N;
        best_NST = NST;
        smem_fold = with;
      }
    }
    for (int NST = 6; NST >= 2 && !best_N; NST--) {
      if (tc_smem_layout(P.nkc, P.a_terms, N, NST, lists, true, false).total <= smem_max) {
        best_N = N;
        best_NST = NST;
      }
    }
  }
  for (int NST = 6; NST >= least && !best_N; NST--) {  // without the ring
    if (tc_smem_layout(P.nkc, P.a_terms, 128, NST, lists, false, false).total <= smem_max) {
      best_N = 128;
      best_NST = NST;
    }
  }
  if (!best_N) return P;
  P.N = best_N;
  P.NST = best_NST;
  P.qtiles = (nq + TC_M - 1) / TC_M;
  P.r_pad = ((nc + 255) / 256) * 256;
  P.rtiles = P.r_pad / P.N;
  P.q_pad = P.qtiles * TC_M;
  // splits: balance waves (one CTA per SM)
  const int smax = std::min(P.rtiles, max_splits > 0 ? max_splits : 16);
  int best_s = 1;
  double best = 1e300;
  for (int s = 1; s <= smax; s++) {
    const long long items = (long long)P.qtiles * s;
    // each split pays a start-up burst before the shared threshold tightens
    const double cost = (double)((items + sms - 1) / sms) / s * (1.0 + 0.03 * s);
    if (cost < best - 1e-12) { best = cost; best_s = s; }
  }
  P.S = best_s;
  P.tiles_per_split = (P.rtiles + P.S - 1) / P.S;
  P.hk = tc_heap_k(k);
  P.smem = tc_smem_layout(P.nkc, P.a_terms, P.N, P.NST, lists, true, false).total;
  P.ringed = P.smem <= smem_max;
  if (!P.ringed)
    P.smem = tc_smem_layout(P.nkc, P.a_terms, P.N, P.NST, lists, false, false).total;
  P.smem_fold = smem_fold;
  // (no log needs more than the quads its part of a split holds, and the room that two chunks want.
  // The entries depend on the splits and on k alone: a serving slot's workspace is allocated once,
  // for the largest of its batches, and short logs end in the brute force: cut to 16 GB in all,
  // 1,000,000 x 131,072, d = 128, k = 128 took 866 ms, and 34.7 s on clusters of sigma 0.02; calls
  // whose logs would take more run in chunks of rows instead)
  P.logcap = std::min(log_entries(std::max(8 * P.kp, 1024), tight),
                      P.tiles_per_split * (P.N / NPART / 4) + LOG_ROOM);
  // workspace: [prepared candidates | query side]
  P.cand_bytes = with_cand ? al256(tc_cand_bytes(nc, d, mode)) : 0;
  size_t off = P.cand_bytes;
  auto take = [&](size_t b) { size_t o = off; off = al256(off + b); return o; };
  P.o_pa = take((size_t)P.q_pad * P.d_pad * elem);
  P.o_pa_lo = P.fmt == 2 ? take((size_t)P.q_pad * P.d_pad * elem) : 0;
  P.o_qn = take((size_t)P.q_pad * 4);
  P.o_qe = take((size_t)P.q_pad * 16);
  P.o_qmx = take((size_t)P.q_pad * 4);
  // NPART logs per (query, split): one per epilogue warp of a lane quarter
  P.o_logcnt = take((size_t)NPART * P.S * nq * 4);
  P.o_proot = take((size_t)NPART * P.S * nq * 4);
  P.o_margin = take((size_t)nq * 4);
  P.o_fbl = take((size_t)nq * 4);
  P.o_fbc = take(16);
  // last: once the re-rank has read the logs, the escalation pass takes their place
  P.log_bytes = (size_t)NPART * P.S * nq * P.logcap * LOG_ENTRY;
  P.o_log = take(P.log_bytes);
  P.bytes = off;
  // Error-bound coefficients. kA: accumulation, charged as truncation on the sum of the products'
  // magnitudes, |q~| |c~| (1 + u)^2 (the rounded factors), over the products and the norm column's
  // MMA, and the FP32 rounding of both centred factors. kB: FP32 rounding of the
  // norm terms. kS: the FP64 distance's own rounding (and the effective norms'). With the norm
  // column its MMA, the last in split BF16 and the first in the others, also adds the three parts of
  // -cn/2 (exact in the input format), whose magnitudes sum to CN / 2; in v = -2w that is twice as
  // much: kC_fold. The final d' = v + qn'
  // rounds once, inside the kB term. The input rounding itself is measured (tc_pack).
  {
    const double D = (double)P.d_pad;
    const double u = P.fmt == 0 || P.fmt == 3 ? std::ldexp(1.0, -11) : std::ldexp(1.0, -8);
    const double n = (P.fmt == 2 ? 3.0 * D : D) + NORM_TERMS;
    const double acc = n * std::ldexp(1.0, -23), last = NORM_TERMS * std::ldexp(1.0, -23);
    P.kA = (float)(acc * (1 + u) * (1 + u) + std::ldexp(1.0, -22));
    P.kB = (float)(1.25 * 3.0 * std::ldexp(1.0, -24) + 1e-12);
    P.kC_fold = (float)(1.25 * ((P.fmt == 2 ? last : acc) + std::ldexp(1.0, -24)) + 1e-12);
    P.kS = (float)(1.25 * (4.0 * d + 32.0) * std::ldexp(1.0, -53));
  }
  P.ok = true;
  return P;
}

// panels in one format: the data panel(s), then the norm panel
static size_t panel_bytes(int r_pad, int d_pad, int fmt) {
  const size_t one = al256((size_t)r_pad * d_pad * (fmt == 0 ? 4 : 2));
  return (fmt == 2 ? 2 * one : one) + al256((size_t)r_pad * tc::NORM_ROW);
}

size_t tc_cand_panel_bytes(int nc, int d, int mode) {
  const CandLayout L = cand_layout(nc, d, mode);
  return panel_bytes(L.r_pad, L.d_pad, L.fmt);
}

// Split BF16 has the narrowest band; a query whose BF16 or TF32 log overflowed runs again in it
// (or, from BF16, in TF32 where the split tiles do not fit).
int tc_escalation_mode(int nq, int nc, int d, int k, int mode, int sms) {
  const int fmt = tc_format_of_mode(mode);
  if (fmt == 2) return 0;
  if (tc_plan_base(nq, nc, d, k, GSKNN_TC_BF16X3, sms, false, 0).ok) return GSKNN_TC_BF16X3;
  if (fmt != 0 && tc_plan_base(nq, nc, d, k, GSKNN_TC_TF32, sms, false, 0).ok)
    return GSKNN_TC_TF32;
  return 0;
}

TcPlan tc_plan(int nq, int nc, int d, int k, int mode, int sms, bool with_cand,
               int max_splits, bool tight) {
  TcPlan P = tc_plan_base(nq, nc, d, k, mode, sms, with_cand, max_splits, tight);
  if (!P.ok) return P;
  P.esc_mode = tc_escalation_mode(nq, nc, d, k, mode, sms);
  if (P.esc_mode) {
    const TcPlan EP = tc_plan_base(nq, nc, d, k, P.esc_mode, sms, false, max_splits, tight);
    P.o_esc = P.o_log;
    size_t off = al256(std::max(P.bytes, P.o_esc + EP.bytes));
    if (with_cand) {  // per-call candidates: their escalation panels live in the workspace
      P.o_ecand = off;
      P.ecand_bytes = panel_bytes(EP.r_pad, EP.d_pad, EP.fmt);
      off = al256(off + P.ecand_bytes);
    }
    P.bytes = off;
  }
  return P;
}

// The escalation pass's candidates: panels, norms and statistics of the second format.
static TcCand escalation_cand(const TcCand &C, const TcPlan &EP, void *pb, void *pb_lo, void *pn) {
  TcCand E = C;
  E.fmt = EP.fmt;
  E.elem = EP.elem;
  E.d_pad = EP.d_pad;
  E.pb = pb;
  E.pb_lo = pb_lo;
  E.pn = pn;
  E.stats = C.estats;
  return E;
}

// Candidates in a double query's band beyond which the CUDA-core kernel is the cheaper way to its
// list. An exact distance of the re-rank costs 5 to 13 pairs of that kernel (B200, ps, d = 8, 32, 100,
// 256: 86, 84, 285, 670 against 16, 12, 31, 53), so a twelfth of the candidates; less where the
// queries are too few to fill the chip (a warp each, or a CTA each). Bands of the whole set, us, CUDA
// cores alone / without the limit / with it: 4,096 x 20,000, d = 32, k = 16, points of scale 1e-20 998
// / 8,061 / 1,376; 5,000 x 50,000, d = 100, unit cube at 1e6 6,037 / 68,192 / 7,060; 16 x 100,000,
// d = 100 650 / 35,158 / 773; 40 x 200,000, d = 32, k = 50 in clusters of 12,500 657 / 3,769 / 1,171.
static int band_limit_of(int nq, int nc, int k, bool cta) {
  const double part = cta ? 0.5 + 0.5 * std::min(1.0, nq / 500.0) : std::min(1.0, nq / 1000.0);
  return (int)std::max(4.0 * k + 256.0, nc / 12.0 * part);
}

// One approximate pass + re-rank: pack the queries (all of them, or on an escalation pass the
// `dQ` queries listed in `rowmap`) and, with `pack_cand`, the candidates C (for the escalation pass
// only if some query is listed); tc_knn in the plan's format; tc_rerank. Queries whose log
// overflowed are appended (as heap rows) to the plan's fallback list, whose count sits at
// base + P.o_fbc.
template <typename T>
static cudaError_t tc_pass(const TcPlan &P, const TcCand &C, bool pack_cand, bool sums, int nq,
                           int d, int k, const T *Xq, const T *Xq2, long long nrows_q,
                           const int *qidx, const int *dQ, const int *rowmap, T *D, int *I,
                           int ldD, char *base, int *status, float *dbg, long long dbg_ld,
                           unsigned long long *counters, cudaStream_t st, TraceHook hook,
                           void *hook_ctx) {
  using namespace tc;
  const bool escalation = dQ != nullptr;
  void *pa = base + P.o_pa;
  void *pa_lo = P.fmt == 2 ? base + P.o_pa_lo : nullptr;
  float *qn = reinterpret_cast<float *>(base + P.o_qn);
  int *fbc = reinterpret_cast<int *>(base + P.o_fbc);
  // tracer brackets; `nk` = kernels of this file launched inside the bracket
  auto mark = [&](const char *name, bool begin, int nk = 0) {
    if (hook) hook(hook_ctx, name, begin, st, nk);
  };
  const char *n_pack = escalation ? "tc_escalate" : "tc_pack";
  const char *n_knn = escalation ? "tc_escalate" : "tc_knn";
  const char *n_rr = escalation ? "tc_escalate" : "tc_rerank";
  PackSide<T> qs{};
  qs.X = Xq;
  qs.X2 = Xq2;
  qs.nrows = nrows_q;
  qs.idx = qidx;
  qs.rowmap = rowmap;
  qs.dcount = dQ;
  qs.count = nq;
  qs.rows_pad = P.q_pad;
  qs.panel = pa;
  qs.panel_lo = pa_lo;
  qs.enorm = qn;
  qs.qe = reinterpret_cast<float4 *>(base + P.o_qe);
  qs.qmx = reinterpret_cast<float *>(base + P.o_qmx);
  qs.Din = D;
  qs.ldD = ldD;
  qs.k = k;
  qs.nroots = NPART * P.S;
  qs.nproot = nq;
  qs.proot = reinterpret_cast<unsigned *>(base + P.o_proot);
  qs.zero = fbc;
  PackSide<T> cs{};
  if (pack_cand) {
    cs = cand_side<T>(C);
    if (escalation) {
      cs.enorm = nullptr;
      cs.gate = dQ;
    }
  }
  mark(n_pack, true);
  cudaError_t e = launch_tc_pack<T>(cs, qs, C, P.fmt, P.d_pad, sums, P.kA, P.kB, P.kS, status, st);
  mark(n_pack, false, 1);
  if (e != cudaSuccess) return e;

  CUtensorMap mA, mAlo, mB, mBlo;
  e = make_panel_map(&mA, pa, P.elem, P.d_pad, P.q_pad, TC_M);
  if (e == cudaSuccess) e = make_panel_map(&mB, C.pb, P.elem, P.d_pad, P.r_pad, P.N);
  if (e != cudaSuccess) return e;
  mAlo = mA;
  mBlo = mB;
  if (P.fmt == 2) {
    e = make_panel_map(&mAlo, pa_lo, P.elem, P.d_pad, P.q_pad, TC_M);
    if (e == cudaSuccess) e = make_panel_map(&mBlo, C.pb_lo, P.elem, P.d_pad, P.r_pad, P.N);
    if (e != cudaSuccess) return e;
  }
  TcParams tp{};
  tp.Q = nq; tp.nkc = P.nkc; tp.ntiles_r = P.rtiles;
  tp.N = P.N; tp.NST = P.NST; tp.logcap = P.logcap;
  tp.a_terms = P.a_terms;
  tp.idesc = idesc_f32acc(P.fmt == 0 ? 2u : P.fmt == 3 ? 0u : 1u, TC_M, P.N);
  tp.fscale = P.fmt == 3 ? C.fscale : nullptr;
  tp.cn = C.cn; tp.qn = qn; tp.qe = qs.qe; tp.qmx = qs.qmx; tp.stats = C.stats;
  tp.log = reinterpret_cast<float4 *>(base + P.o_log);
  tp.logpos = reinterpret_cast<uint32_t *>(tp.log + (size_t)NPART * P.S * nq * P.logcap);
  tp.logcnt = reinterpret_cast<int *>(base + P.o_logcnt);
  tp.proot = qs.proot;
  tp.hk = P.hk;
  tp.W = tc_window(P.S);
  tp.S = P.S;
  tp.margin = reinterpret_cast<float *>(base + P.o_margin);
  tp.status = status;
  tp.dbg = dbg;
  tp.dbg_ld = dbg_ld;
  tp.dbg_ncols = C.nc;
  tp.counters = counters;
  tp.dQ = dQ;
  tp.rowmap = rowmap;
  tp.no_compact = P.esc_mode != 0;
  dim3 grid(P.qtiles, P.S);
  mark(n_knn, true);
  e = launch_tc_knn(P, C.pn, P.r_pad, grid, mA, mAlo, mB, mBlo, tp, st);
  mark(n_knn, false, 1);
  if (e != cudaSuccess) return e;

  RerankParams<T> rp{};
  rp.Q = nq; rp.k = k; rp.S = NPART * P.S; rp.logcap = P.logcap; rp.d = d;
  rp.log = tp.log; rp.logpos = tp.logpos; rp.logcnt = tp.logcnt; rp.margin = tp.margin;
  rp.qn = tp.qn; rp.qmx = tp.qmx; rp.fold = tp.fold; rp.fscale = tp.fscale;
  rp.proot = tp.proot;
  rp.Xq = Xq; rp.Xq2 = Xq2; rp.nrows_q = nrows_q;
  rp.Xc = static_cast<const T *>(C.Xc); rp.Xc2 = static_cast<const T *>(C.Xc2);
  rp.qidx = qidx; rp.cid = C.cid;
  rp.D = D; rp.I = I; rp.ldD = ldD;
  rp.fallback_list = reinterpret_cast<int *>(base + P.o_fbl);
  rp.fallback_count = fbc;
  rp.counters = counters;
  rp.dQ = dQ;
  rp.rowmap = rowmap;
  const int rb = (nq + RR_WARPS - 1) / RR_WARPS;
  // one CTA per query up to four waves of one CTA per SM: 16 queries x 4,096 took 21 us against
  // 40 us with a warp each; at 2,003 queries the warps fill the chip (37 us against 67 us)
  const bool cta = nq <= 4 * P.sms && rp.S <= RC_LOGS;
  rp.limit = band_limit_of(nq, C.nc, k, cta);
  mark(n_rr, true);
  switch (P.kp) {
    case 32: cta ? tc_rerank_cta<T, 1><<<nq, 32 * RR_WARPS, 0, st>>>(rp)
                 : tc_rerank<T, 1><<<rb, 32 * RR_WARPS, 0, st>>>(rp); break;
    case 64: cta ? tc_rerank_cta<T, 2><<<nq, 32 * RR_WARPS, 0, st>>>(rp)
                 : tc_rerank<T, 2><<<rb, 32 * RR_WARPS, 0, st>>>(rp); break;
    case 128: cta ? tc_rerank_cta<T, 4><<<nq, 32 * RR_WARPS, 0, st>>>(rp)
                  : tc_rerank<T, 4><<<rb, 32 * RR_WARPS, 0, st>>>(rp); break;
    case 256: cta ? tc_rerank_cta<T, 8><<<nq, 32 * RR_WARPS, 0, st>>>(rp)
                  : tc_rerank<T, 8><<<rb, 32 * RR_WARPS, 0, st>>>(rp); break;
    default: return cudaErrorInvalidValue;
  }
  e = cudaGetLastError();
  mark(n_rr, false, 1);
  return e;
}

// Exact FP64 brute force for the queries (heap rows) listed at base + P.o_fbl.
static cudaError_t tc_brute(const TcPlan &P, const TcCand &C, int d, int k, const float *Xq,
                            const float *Xq2, long long nrows_q, const int *qidx, float *D,
                            int *I, int ldD, char *base, cudaStream_t st, TraceHook hook,
                            void *hook_ctx,
                            const int *status = nullptr, int *mirror = nullptr) {
  using namespace tc;
  FallbackParams fp{};
  fp.status = status; fp.mirror = mirror;
  fp.k = k; fp.d = d; fp.nc = C.nc; fp.Xq = Xq; fp.Xq2 = Xq2;
  fp.Xc = static_cast<const float *>(C.Xc); fp.Xc2 = static_cast<const float *>(C.Xc2);
  fp.qidx = qidx; fp.cidx = C.cidx; fp.nrows_q = nrows_q; fp.nrows_c = C.nrows_c;
  fp.D = D; fp.I = I; fp.ldD = ldD;
  fp.list = reinterpret_cast<const int *>(base + P.o_fbl);
  fp.count = reinterpret_cast<const int *>(base + P.o_fbc);
  if (hook) hook(hook_ctx, "tc_fallback", true, st, 0);
  switch (P.kp) {
    case 32: tc_fallback<1><<<CHIP_SMS, 256, 0, st>>>(fp); break;
    case 64: tc_fallback<2><<<CHIP_SMS, 256, 0, st>>>(fp); break;
    case 128: tc_fallback<4><<<CHIP_SMS, 256, 0, st>>>(fp); break;
    case 256: tc_fallback<8><<<CHIP_SMS, 256, 0, st>>>(fp); break;
    default: return cudaErrorInvalidValue;
  }
  cudaError_t e = cudaGetLastError();
  if (hook) hook(hook_ctx, "tc_fallback", false, st, 1);
  return e;
}

// The pass in the plan's format, then the escalation: the queries whose log overflowed run again in
// the narrower format against the same candidates (their panels in that format: prepared with the
// candidates, or packed here only when some query overflowed), as a pass over the list of
// overflowed heap rows whose length stays on the device. *list / *count: the heap rows (and their
// number) that overflowed in the last format too.
template <typename T>
static cudaError_t tc_passes(const TcPlan &P, const TcCand &C, bool per_call, int nq, int d, int k,
                             const T *Xq, const T *Xq2, long long nrows_q, const int *qidx, T *D,
                             int *I, int ldD, char *base, int *status, float *dbg,
                             long long dbg_ld, unsigned long long *counters, cudaStream_t st,
                             TraceHook hook, void *hook_ctx, const TcPlan **last, char **last_base,
                             TcPlan *EPout) {
  if (C.fmt != P.fmt || C.d_pad != P.d_pad || C.r_pad != P.r_pad) return cudaErrorInvalidValue;
  *last = &P;
  *last_base = base;
  cudaError_t e = tc_pass<T>(P, C, per_call, per_call, nq, d, k, Xq, Xq2, nrows_q, qidx, nullptr,
                             nullptr, D, I, ldD, base, status, dbg, dbg_ld, counters, st, hook,
                             hook_ctx);
  if (e != cudaSuccess || !P.esc_mode) return e;
  TcPlan &EP = *EPout;
  EP = tc_plan_base(nq, C.nc, d, k, P.esc_mode, P.sms, false, P.max_splits, P.tight);
  void *epb = nullptr, *epb_lo = nullptr, *epn = nullptr;
  bool pack = false;
  if (EP.ok && C.efmt == EP.fmt) {
    epb = C.epb;
    epb_lo = C.epb_lo;
    epn = C.epn;
  } else if (EP.ok && P.ecand_bytes) {
    // the layout of panel_bytes: data panel(s), then the norm panel
    const size_t one = al256((size_t)EP.r_pad * EP.d_pad * EP.elem);
    epb = base + P.o_ecand;
    epb_lo = EP.fmt == 2 ? base + P.o_ecand + one : nullptr;
    epn = base + P.o_ecand + (EP.fmt == 2 ? 2 * one : one);
    pack = true;
  }
  if (!epb) return cudaSuccess;
  const TcCand C2 = escalation_cand(C, EP, epb, epb_lo, epn);
  *last = EPout;
  *last_base = base + P.o_esc;
  return tc_pass<T>(EP, C2, pack, false, nq, d, k, Xq, Xq2, nrows_q, qidx,
                    reinterpret_cast<const int *>(base + P.o_fbc),
                    reinterpret_cast<const int *>(base + P.o_fbl), D, I, ldD, *last_base, status,
                    nullptr, 0, nullptr, st, hook, hook_ctx);
}

// The per-call passes: candidates prepared in the workspace, then tc_passes.
template <typename T>
static cudaError_t tc_call(const TcPlan &P, TcCand *C, int nq, int nc, int d, int k, const T *Xq,
                           const T *Xq2, long long nrows_q, const int *qidx, const T *Xc,
                           const T *Xc2, long long nrows_c, const int *cidx, T *D, int *I, int ldD,
                           void *ws, int *status, float *dbg, long long dbg_ld,
                           unsigned long long *counters, cudaStream_t st, TraceHook hook,
                           void *hook_ctx, const TcPlan **last, char **last_base, TcPlan *EP,
                           bool clear_status) {
  if (P.cand_bytes == 0) return cudaErrorInvalidValue;
  if (hook) hook(hook_ctx, "tc_pack", true, st, 0);
  const cudaError_t e = cand_begin<T>(C, ws, nc, d, tc_mode_of_format(P.fmt), Xc, Xc2, nrows_c,
                                      cidx, clear_status ? status : nullptr, st);
  if (hook) hook(hook_ctx, "tc_pack", false, st, 1);
  if (e != cudaSuccess) return e;
  return tc_passes<T>(P, *C, true, nq, d, k, Xq, Xq2, nrows_q, qidx, D, I, ldD,
                      static_cast<char *>(ws), status, dbg, dbg_ld, counters, st, hook, hook_ctx,
                      last, last_base, EP);
}

cudaError_t tc_run(const TcPlan &P, int nq, int nc, int d, int k, const float *Xq,
                   const float *Xq2, long long nrows_q, const int *qidx, const float *Xc,
                   const float *Xc2, long long nrows_c, const int *cidx, float *D, int *I,
                   int ldD, void *ws, int *status, float *dbg, long long dbg_ld,
                   unsigned long long *counters, cudaStream_t st, TraceHook hook,
                   void *hook_ctx, int *mirror, bool clear_status) {
  TcCand C{};
  const TcPlan *last;
  char *lbase;
  TcPlan EP;
  const cudaError_t e = tc_call<float>(P, &C, nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2,
                                       nrows_c, cidx, D, I, ldD, ws, status, dbg, dbg_ld, counters,
                                       st, hook, hook_ctx, &last, &lbase, &EP, clear_status);
  if (e != cudaSuccess) return e;
  return tc_brute(*last, C, d, k, Xq, Xq2, nrows_q, qidx, D, I, ldD, lbase, st, hook, hook_ctx,
                  status, mirror);
}

cudaError_t tc_run_double(const TcPlan &P, int nq, int nc, int d, int k, const double *Xq,
                          const double *Xq2, long long nrows_q, const int *qidx,
                          const double *Xc, const double *Xc2, long long nrows_c,
                          const int *cidx, double *D, int *I, int ldD, void *ws, int *status,
                          const int **left, const int **nleft, cudaStream_t st, TraceHook hook,
                          void *hook_ctx, bool clear_status) {
  TcCand C{};
  const TcPlan *last;
  char *lbase;
  TcPlan EP;
  const cudaError_t e = tc_call<double>(P, &C, nq, nc, d, k, Xq, Xq2, nrows_q, qidx, Xc, Xc2,
                                        nrows_c, cidx, D, I, ldD, ws, status, nullptr, 0, nullptr,
                                        st, hook, hook_ctx, &last, &lbase, &EP, clear_status);
  if (e != cudaSuccess) return e;
  *left = reinterpret_cast<const int *>(lbase + last->o_fbl);
  *nleft = reinterpret_cast<const int *>(lbase + last->o_fbc);
  return cudaSuccess;
}

cudaError_t tc_run_prepared(const TcPlan &P, const TcCand &C, int nq, int d, int k,
                            const float *Xq, const float *Xq2, long long nrows_q,
                            const int *qidx, float *D, int *I, int ldD, void *ws, int *status,
                            float *dbg, long long dbg_ld, unsigned long long *counters,
                            cudaStream_t st, TraceHook hook, void *hook_ctx) {
  const TcPlan *last;
  char *lbase;
  TcPlan EP;
  const cudaError_t e = tc_passes<float>(P, C, false, nq, d, k, Xq, Xq2, nrows_q, qidx, D, I, ldD,
                                         static_cast<char *>(ws), status, dbg, dbg_ld, counters,
                                         st, hook, hook_ctx, &last, &lbase, &EP);
  if (e != cudaSuccess) return e;
  return tc_brute(*last, C, d, k, Xq, Xq2, nrows_q, qidx, D, I, ldD, lbase, st, hook, hook_ctx);
}

// Escalation panels of a prepared candidate set (kept with it, e.g. a serving engine's
// resident set): the same rows in `mode`'s format, sharing shift, norms and ids.
cudaError_t tc_cand_prepare_escalation(TcCand *C, void *mem, int mode, int *status,
                                       cudaStream_t st) {
  const CandLayout L = cand_layout(C->nc, C->d, mode);
  if (L.r_pad != C->r_pad) return cudaErrorInvalidValue;
  char *b = static_cast<char *>(mem);
  const size_t one = al256((size_t)L.r_pad * L.d_pad * L.elem);
  C->efmt = L.fmt;
  C->epb = b;
  C->epb_lo = L.fmt == 2 ? b + one : nullptr;
  C->epn = b + (L.fmt == 2 ? 2 * one : one);
  tc::PackSide<float> s = cand_side<float>(*C);
  s.panel = C->epb;
  s.panel_lo = C->epb_lo;
  s.npanel = C->epn;
  s.enorm = nullptr;
  s.stats = C->estats;
  return launch_tc_pack<float>(s, tc::PackSide<float>{}, *C, L.fmt, L.d_pad, false, 0.0f, 0.0f,
                               0.0f, status, st);
}

// ------------------------------------------------------------------------------------------
// batching form: leaf panels
// ------------------------------------------------------------------------------------------
namespace tc {
__global__ void iota_kernel(int *a, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    a[i] = (int)i;
}
}  // namespace tc

int tc_leaf_tile(int d, int k, int sms) {
  const TcPlan P = tc_plan_base(256, 256, d, k, GSKNN_TC_BF16X3, sms, false, 1);
  return P.ok ? P.N : 0;
}

TcLeafPlan tc_leaf_plan(long long npts, int rows_cap, int d, int k, int sms, bool tight) {
  using namespace tc;
  TcLeafPlan L{};
  L.ok = false;
  // the tile plan: split BF16, one split, candidate tiles of N (256 where it fits)
  TcPlan P = tc_plan_base(256, 256, d, k, GSKNN_TC_BF16X3, sms, false, 1);
  if (!P.ok || npts <= 0 || rows_cap <= 0 || rows_cap % TC_M != 0) return L;
  L.rows_cap = rows_cap;
  // per-query area for rows_cap rows, one split; smaller logs than the per-call path: a leaf offers
  // a few thousand candidates, of which a part logs about hk (1 + ln(n / hk)) < 5 hk quads (a full
  // log overflows to the leaf brute force), and the room that two chunks want
  P.logcap = 6 * tc_heap_k(k) + 24 + LOG_ROOM;
  if (tight) P.logcap = std::min(P.logcap, log_entries(std::max(2 * P.kp, 256), true));
  P.S = 1;
  P.qtiles = L.rows_cap / TC_M;
  P.q_pad = L.rows_cap;
  size_t off = 0;
  auto take = [&](size_t b) { size_t o = off; off = al256(off + b); return o; };
  const size_t R = (size_t)L.rows_cap;
  L.o_mu = take((size_t)d * 4);
  L.o_fscale = take(8);
  L.o_cpart = take((size_t)CENTER_PARTS * d * 8 + CENTER_SLICES * 4);
  L.o_stats = take(STATS_WORDS * 4);
  L.o_pb = take(R * P.d_pad * 2);
  L.o_pb_lo = take(R * P.d_pad * 2);
  L.o_pn = take(R * NORM_ROW);
  L.o_cn = take(R * 4);
  L.o_cid = take(R * 4);
  L.o_iota = take((size_t)npts * 4);
  P.o_pa = L.o_pb;  // the query panel is the candidate panel
  P.o_pa_lo = L.o_pb_lo;
  P.o_qn = L.o_cn;
  P.o_qe = take(R * 16);
  P.o_qmx = take(R * 4);
  P.o_log = take((size_t)NPART * R * P.logcap * LOG_ENTRY);
  P.o_logcnt = take((size_t)NPART * R * 4);
  P.o_proot = take((size_t)NPART * R * 4);
  P.o_margin = take(R * 4);
  P.o_fbl = take(R * 4);
  P.o_fbc = take(16);
  P.esc_mode = 0;
  P.bytes = off;
  L.bytes = off;
  L.P = P;
  L.ok = true;
  return L;
}

int tc_leaf_tile(const TcLeafPlan &L) { return L.P.N; }

cudaError_t tc_leaf_pass(const TcLeafPlan &L, void *ws, const float *X, const float *X2,
                         long long npts, int d, int k, const int *pidx, int rows,
                         const int4 *qtab, int nqt, const int2 *rtab, float *D, int *I,
                         int ldD, int *status, cudaStream_t st, bool setup,
                         unsigned long long *counters) {
  using namespace tc;
  const TcPlan &P = L.P;
  if (!L.ok || rows > L.rows_cap || rows % P.N != 0 || k > 256) return cudaErrorInvalidValue;
  if (nqt == 0) return cudaSuccess;
  char *base = static_cast<char *>(ws);
  float *mu = reinterpret_cast<float *>(base + L.o_mu);
  unsigned *stats = reinterpret_cast<unsigned *>(base + L.o_stats);
  void *pb = base + L.o_pb, *pb_lo = base + L.o_pb_lo, *pn = base + L.o_pn;
  float *cn = reinterpret_cast<float *>(base + L.o_cn);
  uint32_t *cid = reinterpret_cast<uint32_t *>(base + L.o_cid);
  int *iota = reinterpret_cast<int *>(base + L.o_iota);
  int *fbc = reinterpret_cast<int *>(base + P.o_fbc);
  cudaError_t e = cudaMemsetAsync(stats, 0, STATS_WORDS * 4, st);
  if (e != cudaSuccess) return e;
  TcCand C{};
  C.d = d;
  C.mu = mu;
  C.fscale = reinterpret_cast<float *>(base + L.o_fscale);
  C.part = reinterpret_cast<double *>(base + L.o_cpart);
  C.part_n = reinterpret_cast<int *>(base + L.o_cpart + (size_t)CENTER_PARTS * d * 8);
  if (setup) {
    // once per workspace: the row index map, and the shift (mean of a strided sample of the
    // first panel's rows, padding skipped), which serves every later tree of the same table
    iota_kernel<<<296, 256, 0, st>>>(iota, npts);
    tc_center<float><<<dim3((d + 31) / 32, CENTER_SLICES), 32 * CENTER_WARPS, 0, st>>>(
        X, d, npts, pidx, rows, std::min(rows, CENTER_ROWS), C.part, C.part_n, nullptr, 0,
        nullptr);
  }
  // the panel's rows are candidates and queries at once
  PackSide<float> ps{};
  ps.X = X;
  ps.X2 = X2;
  ps.nrows = npts;
  ps.idx = pidx;
  ps.count = rows;
  ps.rows_pad = rows;
  ps.pad_ok = 1;
  ps.panel = pb;
  ps.panel_lo = pb_lo;
  ps.npanel = pn;
  ps.enorm = cn;
  ps.ids = cid;
  ps.stats = stats;
  ps.qe = reinterpret_cast<float4 *>(base + P.o_qe);
  ps.qmx = reinterpret_cast<float *>(base + P.o_qmx);
  ps.Din = D;
  ps.ldD = ldD;
  ps.k = k;
  ps.nroots = NPART;
  ps.nproot = rows;
  ps.proot = reinterpret_cast<unsigned *>(base + P.o_proot);
  ps.zero = fbc;
  e = launch_tc_pack<float>(PackSide<float>{}, ps, C, 2, P.d_pad, setup, P.kA, P.kB, P.kS, status,
                            st);
  if (e != cudaSuccess) return e;
  CUtensorMap mA, mAlo, mB, mBlo;
  e = make_panel_map(&mA, pb, P.elem, P.d_pad, rows, TC_M);
  if (e == cudaSuccess) e = make_panel_map(&mAlo, pb_lo, P.elem, P.d_pad, rows, TC_M);
  if (e == cudaSuccess) e = make_panel_map(&mB, pb, P.elem, P.d_pad, rows, P.N);
  if (e == cudaSuccess) e = make_panel_map(&mBlo, pb_lo, P.elem, P.d_pad, rows, P.N);
  if (e != cudaSuccess) return e;
  TcParams tp{};
  tp.Q = rows; tp.nkc = P.nkc; tp.ntiles_r = rows / P.N;
  tp.N = P.N; tp.NST = P.NST; tp.logcap = P.logcap;
  tp.a_terms = P.a_terms;
  tp.idesc = idesc_f32acc(1u, TC_M, P.N);
  tp.cn = cn; tp.qn = cn; tp.qe = ps.qe; tp.qmx = ps.qmx; tp.stats = stats;
  tp.log = reinterpret_cast<float4 *>(base + P.o_log);
  tp.logpos = reinterpret_cast<uint32_t *>(tp.log + (size_t)NPART * P.S * rows * P.logcap);
  tp.logcnt = reinterpret_cast<int *>(base + P.o_logcnt);
  tp.proot = reinterpret_cast<unsigned *>(base + P.o_proot);
  tp.hk = P.hk;
  tp.W = tc_window(P.S);
  tp.S = P.S;
  tp.margin = reinterpret_cast<float *>(base + P.o_margin);
  tp.status = status;
  tp.rowmap = pidx;
  tp.qtab = qtab;
  tp.counters = counters;
  e = launch_tc_knn(P, pn, rows, nqt, mA, mAlo, mB, mBlo, tp, st);
  if (e != cudaSuccess) return e;
  RerankParams<float> rp{};
  rp.Q = rows; rp.k = k; rp.S = NPART; rp.logcap = P.logcap; rp.d = d;
  rp.log = tp.log; rp.logpos = tp.logpos; rp.logcnt = tp.logcnt; rp.margin = tp.margin;
  rp.qn = tp.qn; rp.qmx = tp.qmx; rp.fold = tp.fold; rp.fscale = tp.fscale;
  rp.proot = tp.proot;
  rp.Xq = X; rp.Xq2 = X2; rp.nrows_q = npts; rp.Xc = X; rp.Xc2 = X2; rp.qidx = iota;
  rp.cid = cid;
  rp.D = D; rp.I = I; rp.ldD = ldD;
  rp.fallback_list = reinterpret_cast<int *>(base + P.o_fbl);
  rp.fallback_count = fbc;
  rp.rowmap = pidx;
  rp.counters = counters;
  LeafFallbackParams fp{};
  fp.k = k; fp.d = d; fp.N = P.N; fp.X = X; fp.X2 = X2; fp.rowmap = pidx; fp.ids = cid;
  fp.rtab = rtab; fp.D = D; fp.I = I; fp.ldD = ldD; fp.list = rp.fallback_list;
  fp.count = fbc;
  const int rb = (rows + RR_WARPS - 1) / RR_WARPS;
  switch (P.kp) {
    case 32:
      tc_rerank_leaf<1><<<rb, 256, 0, st>>>(rp);
      tc_fallback_leaf<1><<<CHIP_SMS, 256, 0, st>>>(fp);
      break;
    case 64:
      tc_rerank_leaf<2><<<rb, 256, 0, st>>>(rp);
      tc_fallback_leaf<2><<<CHIP_SMS, 256, 0, st>>>(fp);
      break;
    case 128:
      tc_rerank_leaf<4><<<rb, 256, 0, st>>>(rp);
      tc_fallback_leaf<4><<<CHIP_SMS, 256, 0, st>>>(fp);
      break;
    case 256:
      tc_rerank_leaf<8><<<rb, 256, 0, st>>>(rp);
      tc_fallback_leaf<8><<<CHIP_SMS, 256, 0, st>>>(fp);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace gsknn
