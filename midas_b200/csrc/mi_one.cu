// mi_one.cu -- kernel (b) for a few frames: the run, CSR and MMA encodings' sums, thread per bin.
//
// The batched kernels' lanes are frames: one frame leaves 31 of 32 lanes idle, and their cost is
// per pass over the map.  Here a lane is a bin.  A bin's terms {pixel, weight} are the ones of
// the plan's tiles in the order in which the batched kernel adds them, with the ends of its
// unit partials marked, so every FP64 sum, every rounding of a partial to FP32 and the scaling
// are the batched kernel's: a frame's cake and lineouts are the same bits on either path, and a
// pixel or dark that is not finite reaches the bins whose terms hold it on both.
//
// MMA plans: the terms carry the fixed-point weights, the sums are exact 64-bit integers and are
// scaled as the tensor-core kernel's epilogue scales them: the same bits again.
//
// Layout: slices of 32 neighbouring bins as in the plain path (PlainLayout): step k holds term k
// of each bin that has one, side by side, nothing padded, 8 B a term.  It is made on the device
// from the tile blobs when the plan is.
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "mi_internal.h"

namespace mi {

constexpr int kPmFrames = 8;                // frames of a pixel side by side
static_assert(kOneChunk <= kPmFrames, "the bin results hold eight frames a bin");
constexpr uint32_t kOneEnd = 0x80000000u;   // the term ends a unit partial

// The terms of one bin in summing order.  Run encoding: the units of the bin's strip, records in
// order, the record's weight for the bin's row where it is not zero.
struct OneTerms {
  const uint8_t *blob;
  TileHdr h;
  int enc, G, L, i, s;          // row and strip (column) in the tile
  uint32_t o_rsp, o_up, o_lc, o_w;
  int u, u_end, j, j1, q;       // unit, its end; record, end of its range; rs of the record
  __device__ void open(const uint8_t *b, int enc_, int G_, int L_, int row, int col) {
    blob = b;
    enc = enc_;
    G = G_;
    L = L_;
    h = *(const TileHdr *)blob;
    i = row;
    s = col;
    uint32_t t0, t1, t2;
    if (enc == MI_ENC_RUNS) {
      runs_blob_layout(h.nb, h.n_cols, h.nnz, h.n_u, G, L, &o_rsp, &t0, &t1, &o_up, &o_lc, &o_w);
      const uint32_t st = ((const uint32_t *)(blob + kRunUnitsOff + kRunWarps * 8))[s];
      u = (int)(st & 0xFFFF) - 1;
      u_end = u + 1 + (int)(st >> 16);
      j = j1 = 0;
    } else {
      uint32_t o_rp;
      blob_layout(h.nb, h.nnz, h.n_u, &o_rp, &t0, &t1, &o_up, &o_lc, &o_w, &t2);
      const uint32_t *rp = (const uint32_t *)(blob + o_rp) + i * h.n_cols + s;
      j = (int)rp[0];
      j1 = (int)rp[1];
    }
  }
  // the next term; false when there is none.  new_unit: the term is the first of its unit
  __device__ bool next(uint32_t *pix, float *w, bool *new_unit) {
    const uint16_t *lcol = (const uint16_t *)(blob + o_lc);
    const uint32_t *upix = (const uint32_t *)(blob + o_up);
    *new_unit = false;
    if (enc != MI_ENC_RUNS) {
      if (j >= j1) return false;
      *pix = upix[lcol[j]];
      *w = ((const float *)(blob + o_w))[j];
      ++j;
      return true;
    }
    const int NRS = G - L + 2;
    const uint16_t *rp = (const uint16_t *)(blob + o_rsp) + s * NRS;
    const int q0 = max(0, i - L + 1), q1 = min(i, G - L);   // records whose rows cover row i
    for (;;) {
      while (j >= j1) {
        if (++u >= u_end) return false;
        const uint16_t *ud = (const uint16_t *)(blob + kRunUnitsOff) + 4 * u;
        j = max((int)ud[1], (int)rp[q0]);
        j1 = min((int)ud[2], (int)rp[q1 + 1]);
        q = q0;
        *new_unit = true;
      }
      while (j >= (int)rp[q + 1]) ++q;
      const float v = ((const float *)(blob + o_w))[(int64_t)j * L + (i - q)];
      const int jj = j++;
      if (v != 0.0f) {
        *pix = upix[lcol[jj]];
        *w = v;
        return true;
      }
    }
  }
};

struct OneBuild {
  PlainLayout g;
  const TileRef *tiles;
  const uint8_t *blobs;
  int32_t *tile_of_bin;
  int32_t *cnt;
  int64_t *slice_n;
  const int64_t *slice_ptr;
  uint2 *terms;
  double *scale;
  const int32_t *xc_pix;    // MMA encoding: pixel of a compact index
  const int32_t *span_lo, *row_off;   // panel plans: the terms name compact indices
  int ny;
  int n_tiles, enc, G, L;
};

__global__ void k_one_tiles(OneBuild a) {
  const int t = blockIdx.x;
  const TileHdr h = *(const TileHdr *)(a.blobs + a.tiles[t].off);
  for (int b = threadIdx.x; b < h.nb; b += blockDim.x)
    a.tile_of_bin[(int64_t)(h.r0 + b / h.n_cols) * a.g.n_eta + h.e0 + b % h.n_cols] = t;
}

__device__ inline bool one_open(const OneBuild &a, int64_t b, OneTerms *it) {
  if (b < 0) return false;
  const uint8_t *blob = a.blobs + a.tiles[a.tile_of_bin[b]].off;
  const TileHdr h = *(const TileHdr *)blob;
  it->open(blob, a.enc, a.G, a.L, (int)(b / a.g.n_eta) - h.r0, (int)(b % a.g.n_eta) - h.e0);
  return true;
}

__global__ void k_one_count(OneBuild a) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= a.g.n_slices) return;
  const int64_t b = plain_bin(a.g, s, lane);
  OneTerms it;
  int n = 0;
  if (one_open(a, b, &it)) {
    uint32_t pix;
    float w;
    bool first;
    while (it.next(&pix, &w, &first)) ++n;
  }
  a.cnt[s * 32 + lane] = n;
  int64_t t = n;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) a.slice_n[s] = t;
}

__global__ void k_one_fill(OneBuild a) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= a.g.n_slices) return;
  const int64_t b = plain_bin(a.g, s, lane);
  const int n = a.cnt[s * 32 + lane];
  int64_t at = a.slice_ptr[s];
  OneTerms it;
  uint32_t pix = 0;
  float w = 0.0f;
  bool first = false, more = one_open(a, b, &it);
  if (more) {
    uint32_t o0, o1, o2, o3, o4, o5, o6;
    if (a.enc == MI_ENC_RUNS) runs_blob_layout(it.h.nb, it.h.n_cols, it.h.nnz, it.h.n_u, a.G, a.L, &o0, &o1, &o2, &o3, &o4, &o5);
    else blob_layout(it.h.nb, it.h.nnz, it.h.n_u, &o0, &o1, &o2, &o3, &o4, &o5, &o6);
    a.scale[b] = ((const double *)(it.blob + o1))[it.i * it.h.n_cols + it.s];
    more = it.next(&pix, &w, &first);
  }
  for (int k = 0; __any_sync(0xffffffffu, k < n); ++k) {
    const int64_t o = plain_step(k < n, lane, at);
    if (k >= n) continue;
    if (a.row_off) {
      const int z = (int)(pix / (uint32_t)a.ny);
      pix = (uint32_t)(a.row_off[z] + (int)(pix - (uint32_t)z * (uint32_t)a.ny) - a.span_lo[z]);
    }
    uint2 t = make_uint2(pix, __float_as_uint(w));
    more = it.next(&pix, &w, &first);
    if (a.enc == MI_ENC_RUNS && (!more || first)) t.x |= kOneEnd;
    a.terms[o] = t;
  }
}

// MMA encoding: a tile's words, each up to four terms of one bin.  The sums are exact integers, so
// the order of a bin's terms is free: a term takes the next place of its bin.
__device__ __forceinline__ int64_t mma_bin(const PlainLayout &g, const MmaHdr &h, int n) {
  const int row = n / kMmaCols, col = n % kMmaCols;
  return row < h.n_rows && col < h.n_cols ? (int64_t)(h.r0 + row) * g.n_eta + h.e0 + col : -1;
}
// slice and lane of a bin (the inverse of plain_bin)
__device__ __forceinline__ int64_t plain_slot(const PlainLayout &g, int64_t b) {
  const int64_t per_row = (g.n_eta + (1 << g.ee) - 1) >> g.ee, r = b / g.n_eta, e = b % g.n_eta;
  const int rr = 32 >> g.ee;
  return ((r / rr) * per_row + (e >> g.ee)) * 32 + (r % rr << g.ee) + (e & ((1 << g.ee) - 1));
}

template <bool FILL>
__global__ void __launch_bounds__(128) k_one_mma(OneBuild a) {
  __shared__ int32_t s_n[kMmaN];
  const uint8_t *blob = a.blobs + a.tiles[blockIdx.x].off;
  const MmaHdr h = *(const MmaHdr *)blob;
  const MmaBlob B = mma_blob_layout(h.n_k, h.n_runs, h.n_terms);
  const uint2 *runs = (const uint2 *)(blob + B.runs);
  const uint32_t *rptr = (const uint32_t *)(blob + B.run_ptr), *sp = (const uint32_t *)(blob + B.step_ptr);
  const uint4 *wpl = (const uint4 *)(blob + B.wpl);
  const uint16_t *widx = (const uint16_t *)(blob + B.widx);
  for (int n = threadIdx.x; n < kMmaN; n += blockDim.x) {
    s_n[n] = 0;
    const int64_t b = mma_bin(a.g, h, n);
    if (!FILL && b >= 0) a.tile_of_bin[b] = (int)blockIdx.x;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < h.n_terms; t += blockDim.x) {
    const int n = widx[t] >> 3;
    const uint4 wv = wpl[t];
    int lo = 0, hi = h.n_k - 1;          // the word's K step
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sp[mid] <= (uint32_t)t) lo = mid;
      else hi = mid - 1;
    }
    for (int c = 0; c < 4; ++c) {
      const uint32_t dg = ((wv.x >> (8 * c)) & 0xFFu) | (((wv.y >> (8 * c)) & 0xFFu) << 8) |
                          (((wv.z >> (8 * c)) & 0xFFu) << 16) | (((wv.w >> (8 * c)) & 0xFFu) << 24);
      if (dg == 0u) continue;
      const int k = atomicAdd(&s_n[n], 1);
      if constexpr (FILL) {
        const uint32_t kk = (widx[t] & 7u) * 4u + (uint32_t)c;   // K slot; its pixel: the run that covers it
        uint32_t px = 0;
        for (uint32_t r = rptr[lo]; r < rptr[lo + 1]; ++r) {
          const uint32_t k0 = runs[r].y & 0xFFu, len = runs[r].y >> 8;
          if (kk >= k0 && kk < k0 + len) px = (uint32_t)a.xc_pix[runs[r].x + (kk - k0)];
        }
        const int64_t slot = plain_slot(a.g, mma_bin(a.g, h, n)), s = slot >> 5;
        const int lane = (int)(slot & 31);
        int64_t o = a.slice_ptr[s];
        for (int l = 0; l < 32; ++l) {
          const int m = a.cnt[s * 32 + l];
          o += min(m, k) + (l < lane && m > k ? 1 : 0);
        }
        a.terms[o] = make_uint2(px, (uint32_t)(int32_t)mma_digits_value(dg));
      }
    }
  }
  if constexpr (!FILL) {
    __syncthreads();
    for (int n = threadIdx.x; n < kMmaN; n += blockDim.x) {
      const int64_t b = mma_bin(a.g, h, n);
      if (b >= 0) a.cnt[plain_slot(a.g, b)] = s_n[n];
    }
  }
}

__global__ void k_one_slices(OneBuild a) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= a.g.n_slices) return;
  int64_t t = a.cnt[s * 32 + lane];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) a.slice_n[s] = t;
}

struct OneArgs {
  PlainLayout g;
  const uint2 *terms;
  const int32_t *cnt;
  const int64_t *slice_ptr;
  const double *scale;
  const void *frames;
  int64_t stride;
  const float *dark;        // null: none
  float *cake;              // [F][n_bins] or null
  double *res;              // [F / 8][n_bins][8] for the lineouts, or null
  int64_t n_bins;
  int F, round_res;         // round_res: the lineouts take the rounded bin results (CSR encoding)
  const int32_t *tile_of_bin;   // MMA encoding: where a bin's factor and dark term are
  const TileRef *tiles;
  const uint8_t *blobs;
};

// NF frames per pass over the map, U terms in flight per lane and as many fetched ahead.  Bounded by
// the gathers' latency and issue together (one 2048^2 gradient frame: issue slots 65 % busy, L1 57, DRAM
// 43, at 41 % of the warps) and at few bins by the latency alone (1024^2, 71,280 bins: 46, 35, 18 % at
// 19 % of the warps).  One frame, cake only, where the run kernel took 298, 936, 1038 and
// 1525 us: 33, 48, 67 and 112 us (1024^2, 495 x 45; 2048^2, 990 x 72; 1980 x 180 gradient; 2880^2,
// 3960 x 360 gradient, 308 MB of terms).
// INT (MMA encoding): integer weights, exact integer sums, the kernel's scaling.
template <typename T, int NF, int U, bool INT>
__global__ void __launch_bounds__(128) k_one(OneArgs a) {
  using Acc = typename std::conditional<INT, long long, double>::type;
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.g.n_slices) return;
  const int64_t s = a.g.n_slices - 1 - i;   // outer rings hold more terms: they start first
  const int64_t b = plain_bin(a.g, s, lane);
  const int n = a.cnt[s * 32 + lane];
  int n_max = n;
  for (int o = 16; o > 0; o >>= 1) n_max = max(n_max, __shfl_xor_sync(0xffffffffu, n_max, o));
  const int64_t first = a.slice_ptr[s];
  int64_t at = first;
  const int f0 = (int)blockIdx.y * NF;
  const T *img[NF];
  Acc acc[NF];
  double tot[NF];
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    img[q] = (const T *)a.frames + (int64_t)min(f0 + q, a.F - 1) * a.stride;
    acc[q] = 0;
    tot[q] = 0.0;
  }
  uint2 t[U];
  if (n_max > 0) plain_load<uint2, U>(a.terms, first, 0, n, lane, at, t);
  for (int k = 0; k < n_max; k += U) {
    uint2 tn[U];
    if (k + U < n_max) plain_load<uint2, U>(a.terms, first, k + U, n, lane, at, tn);
    T raw[U][NF];
    float d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t p = t[u].x & ~kOneEnd;
#pragma unroll
      for (int q = 0; q < NF; ++q) raw[u][q] = __ldg(img[q] + p);
      d[u] = !INT && a.dark ? __ldg(a.dark + p) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = k + u < n;
      if constexpr (INT) {
        const long long w = in ? (long long)(int32_t)t[u].y : 0;
#pragma unroll
        for (int q = 0; q < NF; ++q) acc[q] += w * (long long)(int32_t)raw[u][q];
        continue;
      }
      const double w = (double)__uint_as_float(t[u].y);
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        const double x = fma(w, (double)((float)raw[u][q] - d[u]), (double)acc[q]);
        acc[q] = in ? (Acc)x : acc[q];
      }
      if (in && (t[u].x & kOneEnd)) {
#pragma unroll
        for (int q = 0; q < NF; ++q) {
          tot[q] += (double)(float)acc[q];
          acc[q] = 0.0;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = tn[u];
  }
  if (b < 0) return;
  double sc, dk = 0.0;
  if constexpr (INT) {
    const uint8_t *blob = a.blobs + a.tiles[a.tile_of_bin[b]].off;
    const MmaHdr h = *(const MmaHdr *)blob;
    const int m = ((int)(b / a.g.n_eta) - h.r0) * kMmaCols + (int)(b % a.g.n_eta) - h.e0;
    sc = ((const double *)(blob + kMmaBinsOff))[m];
    dk = ((const double *)(blob + kMmaBinsOff))[kMmaN + m];
  } else {
    sc = a.scale[b];
  }
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    if (f0 + q >= a.F) break;
    double o;
    if constexpr (INT) o = fma(sc, __ll2double_rn(acc[q]), -dk);
    else o = (tot[q] + (double)acc[q]) * sc;   // one of the two is zero
    const int64_t at_bin = (int64_t)(f0 + q) * a.n_bins + b;
    if (a.cake) a.cake[at_bin] = (float)o;
    if (a.res) a.res[b * kPmFrames + f0 + q] = a.round_res ? (double)(float)o : o;   // F <= kOneChunk = 8
  }
}

// ---- many frames, eight to a 32-byte sector
//
// Beyond a few frames the gathers bound k_one: a lane's pixels lie in different lines whatever a
// line brings.  Here eight frames of a pixel lie side by side as fp32 minus the dark (one
// sector), so a gather brings eight values and a term is read once for them.  Bounded by
// the gathers' latency at few warps (1475 x 1679 int32, 790 x 72 bins, 50 frames: 317 us for 29 M
// gathers, 2.9 TB/s from L2; 162 registers leave 17 % of the warps, with L1 58 % busy, L2 30, issue 22)
// and by the staging pass's bytes (150 us, DRAM 65 % busy).  50 such frames with lineouts took 1078 us
// through the 64-frame rows and the run kernel, 800 through k_one; 534 here.
//
// k_pm writes them: a thread per pixel of a span, eight coalesced loads, one 32-byte store.
template <typename T>
__global__ void __launch_bounds__(256) k_pm(const T *__restrict__ frames, int64_t stride, int F, int ny, int z_off,
                                            int ny_v, const float *__restrict__ dark,
                                            const XcChunk *__restrict__ chunks, float *__restrict__ pm, int64_t n_px,
                                            int compact) {
  const XcChunk ch = chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.n) return;
  const int f0 = (int)blockIdx.y * kPmFrames;
  const int64_t o = (int64_t)(ch.z - z_off) * ny + ch.y0 + threadIdx.x;
  const int64_t v = (int64_t)ch.z * ny_v + ch.y0 + threadIdx.x;
  T raw[kPmFrames];
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) raw[q] = f0 + q < F ? __ldg(frames + (int64_t)(f0 + q) * stride + o) : (T)0;
  const float d = __ldg(dark + v);
  float x[kPmFrames];
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) x[q] = f0 + q < F ? (float)raw[q] - d : 0.0f;
  const int64_t at = compact ? (int64_t)ch.c0 + threadIdx.x : v;
  float4 *dst = (float4 *)(pm + ((int64_t)blockIdx.y * n_px + at) * kPmFrames);
  dst[0] = make_float4(x[0], x[1], x[2], x[3]);
  dst[1] = make_float4(x[4], x[5], x[6], x[7]);
}

// the same for MMA plans: eight raw counts of 8/16-bit frames, 16 bytes a pixel (4 frames of 2048^2
// gradient: 186 us through k_one, 116 with these; the sums L1 70 % busy, issue 53, at 40 % of the warps)
template <typename T>
__global__ void __launch_bounds__(256) k_pm16(const T *__restrict__ frames, int64_t stride, int F, int ny,
                                              const XcChunk *__restrict__ chunks, uint4 *__restrict__ pm, int64_t n_px) {
  const XcChunk ch = chunks[blockIdx.x];
  if ((int)threadIdx.x >= ch.n) return;
  const int f0 = (int)blockIdx.y * kPmFrames;
  const int64_t o = (int64_t)ch.z * ny + ch.y0 + threadIdx.x;
  uint32_t x[kPmFrames];
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) x[q] = f0 + q < F ? (uint32_t)__ldg(frames + (int64_t)(f0 + q) * stride + o) : 0u;
  pm[(int64_t)blockIdx.y * n_px + o] =
      make_uint4(x[0] | (x[1] << 16), x[2] | (x[3] << 16), x[4] | (x[5] << 16), x[6] | (x[7] << 16));
}

// a bin's integer sums of eight frames -> cake and results (MMA plans)
template <int U>
__global__ void __launch_bounds__(128) k_one_pm16(OneArgs a, const uint4 *pm, int64_t n_px) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.g.n_slices) return;
  const int64_t s = a.g.n_slices - 1 - i;
  const int64_t b = plain_bin(a.g, s, lane);
  const int n = a.cnt[s * 32 + lane];
  int n_max = n;
  for (int o = 16; o > 0; o >>= 1) n_max = max(n_max, __shfl_xor_sync(0xffffffffu, n_max, o));
  const int64_t first = a.slice_ptr[s];
  int64_t at = first;
  const uint4 *src = pm + (int64_t)blockIdx.y * n_px;
  long long acc[kPmFrames];
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) acc[q] = 0;
  uint2 t[U];
  if (n_max > 0) plain_load<uint2, U>(a.terms, first, 0, n, lane, at, t);
  for (int k = 0; k < n_max; k += U) {
    uint2 tn[U];
    if (k + U < n_max) plain_load<uint2, U>(a.terms, first, k + U, n, lane, at, tn);
    uint4 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = __ldg(src + t[u].x);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long w = k + u < n ? (long long)(int32_t)t[u].y : 0;
      const uint32_t v[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        acc[2 * q] += w * (long long)(int32_t)(v[q] & 0xFFFFu);
        acc[2 * q + 1] += w * (long long)(int32_t)(v[q] >> 16);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = tn[u];
  }
  if (b < 0) return;
  const uint8_t *blob = a.blobs + a.tiles[a.tile_of_bin[b]].off;
  const MmaHdr h = *(const MmaHdr *)blob;
  const int m = ((int)(b / a.g.n_eta) - h.r0) * kMmaCols + (int)(b % a.g.n_eta) - h.e0;
  const double sc = ((const double *)(blob + kMmaBinsOff))[m], dk = ((const double *)(blob + kMmaBinsOff))[kMmaN + m];
  const int f0 = (int)blockIdx.y * kPmFrames;
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) {
    if (f0 + q >= a.F) break;
    const double o = fma(sc, __ll2double_rn(acc[q]), -dk);
    if (a.cake) a.cake[(int64_t)(f0 + q) * a.n_bins + b] = (float)o;
    if (a.res) a.res[((int64_t)blockIdx.y * a.n_bins + b) * kPmFrames + q] = o;
  }
}

template <int U>
__global__ void __launch_bounds__(128) k_one_pm(OneArgs a, const float *pm, int64_t n_px) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.g.n_slices) return;
  const int64_t s = a.g.n_slices - 1 - i;
  const int64_t b = plain_bin(a.g, s, lane);
  const int n = a.cnt[s * 32 + lane];
  int n_max = n;
  for (int o = 16; o > 0; o >>= 1) n_max = max(n_max, __shfl_xor_sync(0xffffffffu, n_max, o));
  const int64_t first = a.slice_ptr[s];
  int64_t at = first;
  const float4 *src = (const float4 *)(pm + (int64_t)blockIdx.y * n_px * kPmFrames);
  double acc[kPmFrames], tot[kPmFrames];
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) acc[q] = tot[q] = 0.0;
  uint2 t[U];
  if (n_max > 0) plain_load<uint2, U>(a.terms, first, 0, n, lane, at, t);
  for (int k = 0; k < n_max; k += U) {
    uint2 tn[U];
    if (k + U < n_max) plain_load<uint2, U>(a.terms, first, k + U, n, lane, at, tn);
    float4 x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float4 *r = src + 2 * (int64_t)(t[u].x & ~kOneEnd);
      x[u][0] = __ldg(r);
      x[u][1] = __ldg(r + 1);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k + u >= n) break;
      const double w = (double)__uint_as_float(t[u].y);
      const float v[kPmFrames] = {x[u][0].x, x[u][0].y, x[u][0].z, x[u][0].w,
                                  x[u][1].x, x[u][1].y, x[u][1].z, x[u][1].w};
#pragma unroll
      for (int q = 0; q < kPmFrames; ++q) acc[q] = fma(w, (double)v[q], acc[q]);
      if (t[u].x & kOneEnd) {
#pragma unroll
        for (int q = 0; q < kPmFrames; ++q) {
          tot[q] += (double)(float)acc[q];
          acc[q] = 0.0;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = tn[u];
  }
  if (b < 0) return;
  const double sc = a.scale[b];
  const int f0 = (int)blockIdx.y * kPmFrames;
#pragma unroll
  for (int q = 0; q < kPmFrames; ++q) {
    if (f0 + q >= a.F) break;
    const double o = (tot[q] + acc[q]) * sc;
    if (a.cake) a.cake[(int64_t)(f0 + q) * a.n_bins + b] = (float)o;
    if (a.res) a.res[((int64_t)blockIdx.y * a.n_bins + b) * kPmFrames + q] = o;
  }
}

// Lineout partials of the items' rows from the bin results, in the batched kernels' order: a
// tile's columns in order, then the tiles.  One thread per (item, row, frame of eight): the eight
// frames of a bin lie side by side, and share the walk over the tiles.
__global__ void k_one_partials(const WorkItem *items, int n_items, const TileRef *tiles, const uint8_t *blobs, int enc,
                               int G, int L, int rows, const double *res, int64_t n_bins, int n_r, int n_eta,
                               int n_slots, int F, double *partial) {
  const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kPmFrames;
  const int q = threadIdx.x % kPmFrames;
  const int64_t f = (int64_t)blockIdx.y * kPmFrames + q;
  if (t >= (int64_t)n_items * rows || f >= F) return;
  const WorkItem it = items[t / rows];
  const int r = it.r0 + (int)(t % rows);
  if (r >= it.r0 + it.n_rows) return;
  const double *row = res + ((int64_t)blockIdx.y * n_bins + (int64_t)r * n_eta) * kPmFrames + q;
  double paw = 0.0, psm = 0.0;
  for (int k = it.tile_begin; k < it.tile_end; ++k) {
    const uint8_t *blob = blobs + tiles[k].off;
    if (enc == MI_ENC_MMA) {
      const MmaHdr h = *(const MmaHdr *)blob;
      if (r < h.r0 || r >= h.r0 + h.n_rows) continue;
      const float *lw = (const float *)(blob + kMmaBinsOff + 16 * kMmaN) + (r - h.r0) * kMmaCols;
      double rw[kMmaCols], rs[kMmaCols];
#pragma unroll
      for (int c = 0; c < kMmaCols; ++c) {
        const double o = c < h.n_cols ? row[(int64_t)(h.e0 + c) * kPmFrames] : 0.0;
        const float l = lw[c];
        rw[c] = o * (double)l;
        rs[c] = (l > 0.0f) ? o : 0.0;
      }
      paw += (rw[0] + rw[1]) + (rw[2] + rw[3]);
      psm += (rs[0] + rs[1]) + (rs[2] + rs[3]);
      continue;
    }
    const TileHdr h = *(const TileHdr *)blob;
    if (r < h.r0 || r >= h.r0 + h.n_rows) continue;
    uint32_t o0, o1, o_lw, o3, o4, o5, o6;
    if (enc == MI_ENC_RUNS) runs_blob_layout(h.nb, h.n_cols, h.nnz, h.n_u, G, L, &o0, &o1, &o_lw, &o3, &o4, &o5);
    else blob_layout(h.nb, h.nnz, h.n_u, &o0, &o1, &o_lw, &o3, &o4, &o5, &o6);
    const float *lw = (const float *)(blob + o_lw) + (r - h.r0) * h.n_cols;
    double saw = 0.0, ssm = 0.0;
    for (int c = 0; c < h.n_cols; ++c) {
      const double o = row[(int64_t)(h.e0 + c) * kPmFrames];
      const float l = lw[c];
      saw += o * (double)l;
      ssm += (l > 0.0f) ? o : 0.0;
    }
    paw += saw;
    psm += ssm;
  }
  double *dst = partial + ((f * n_r + r) * n_slots + it.slot) * 2;
  dst[0] = paw;
  dst[1] = psm;
}

static int launch_one_partials(const Plan *p, const double *res, int F, double *partial, cudaStream_t s) {
  const int rows = p->encoding == MI_ENC_MMA ? kMmaRows : p->lim.rows;
  const int64_t n = (int64_t)p->n_items * rows * kPmFrames;
  k_one_partials<<<dim3((unsigned)((n + 127) / 128), (unsigned)((F + kPmFrames - 1) / kPmFrames)), 128, 0, s>>>(
      p->d_items, p->n_items, p->d_tiles, p->d_blobs, p->encoding, p->run_g, p->run_l, rows, res, p->n_bins, p->n_r,
      p->n_eta, p->n_slots, F, partial);
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}

int build_one(Plan *p, size_t *acct) {
  p->one = plain_layout(p->n_r, p->n_eta);
  const PlainLayout &g = p->one;
  if (p->n_tiles == 0 || p->encoding == MI_ENC_MMAD) return MI_OK;
  const bool mma = p->encoding == MI_ENC_MMA;
  cudaStream_t st = nullptr;
  MI_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  std::vector<void *> tmp;
  auto temp = [&](void **q, size_t bytes) {
    cudaError_t e = cudaMallocAsync(q, std::max<size_t>(bytes, 16), st);
    if (e == cudaSuccess) tmp.push_back(*q);
    return e;
  };
  auto keep = [&](void **q, size_t bytes) {
    *acct += std::max<size_t>(bytes, 16);
    return cudaMalloc(q, std::max<size_t>(bytes, 16));
  };
  auto build = [&]() -> int {
    MI_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // the blobs' copies (pageable) have arrived
    OneBuild a{};
    a.g = g;
    a.tiles = p->d_tiles;
    a.blobs = p->d_blobs;
    a.n_tiles = p->n_tiles;
    a.enc = p->encoding;
    a.G = p->run_g;
    a.L = p->run_l;
    if (mma) {
      MI_CUDA(keep((void **)&p->d_one_tile, sizeof(int32_t) * p->n_bins));
      a.tile_of_bin = p->d_one_tile;
    } else {
      MI_CUDA(temp((void **)&a.tile_of_bin, sizeof(int32_t) * p->n_bins));
    }
    a.xc_pix = p->d_xc_pix;
    if (p->panels.size() > 1) {
      a.span_lo = p->d_span_lo;
      a.row_off = p->d_row_off;
      a.ny = p->ny;
    }
    MI_CUDA(temp((void **)&a.slice_n, sizeof(int64_t) * g.n_slices));
    MI_CUDA(keep((void **)&p->d_one_cnt, sizeof(int32_t) * 32 * g.n_slices));
    MI_CUDA(keep((void **)&p->d_one_ptr, sizeof(int64_t) * g.n_slices));
    if (!mma) MI_CUDA(keep((void **)&p->d_one_scale, sizeof(double) * p->n_bins));
    // the bin results live in the pixel-major buffer, which this path leaves alone, where it is
    // large enough
    const size_t res = sizeof(double) * p->n_bins * kOneChunk;
    p->one_res_in_xc = p->n_xc * kXcRowBytes >= (int64_t)res;
    if (!p->one_res_in_xc) MI_CUDA(keep((void **)&p->d_one_res, res));
    a.cnt = p->d_one_cnt;
    a.scale = p->d_one_scale;
    const unsigned blocks = (unsigned)((g.n_slices * 32 + 127) / 128);
    if (mma) {
      MI_CUDA(cudaMemsetAsync(p->d_one_cnt, 0, sizeof(int32_t) * 32 * g.n_slices, st));
      k_one_mma<false><<<(unsigned)p->n_tiles, 128, 0, st>>>(a);
      MI_CUDA(cudaGetLastError());
      k_one_slices<<<blocks, 128, 0, st>>>(a);
    } else {
      k_one_tiles<<<(unsigned)p->n_tiles, 128, 0, st>>>(a);
      MI_CUDA(cudaGetLastError());
      k_one_count<<<blocks, 128, 0, st>>>(a);
    }
    MI_CUDA(cudaGetLastError());
    std::vector<int64_t> n(g.n_slices);
    MI_CUDA(cudaMemcpyAsync(n.data(), a.slice_n, sizeof(int64_t) * g.n_slices, cudaMemcpyDeviceToHost, st));
    MI_CUDA(cudaStreamSynchronize(st));
    int64_t total = 0;
    for (int64_t &v : n) {
      const int64_t c = v;
      v = total;
      total += c;
    }
    MI_CUDA(cudaMemcpyAsync(p->d_one_ptr, n.data(), sizeof(int64_t) * g.n_slices, cudaMemcpyHostToDevice, st));
    MI_CUDA(keep((void **)&p->d_one_terms, sizeof(uint2) * total));
    a.slice_ptr = p->d_one_ptr;
    a.terms = p->d_one_terms;
    if (mma) k_one_mma<true><<<(unsigned)p->n_tiles, 128, 0, st>>>(a);
    else k_one_fill<<<blocks, 128, 0, st>>>(a);
    MI_CUDA(cudaGetLastError());
    MI_CUDA(cudaStreamSynchronize(st));
    return MI_OK;
  };
  const int rc = build();
  for (void *q : tmp) cudaFreeAsync(q, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return rc;
}

template <typename T, bool INT>
static int launch_one_t(Plan *p, const OneArgs &a, cudaStream_t s) {
  const unsigned bx = (unsigned)((p->one.n_slices * 32 + 127) / 128);
  const bool deep = p->one.n_slices < kPlainDeep * (int64_t)std::max(p->n_sms, 1);
  if (a.F == 1) {
    if (deep) k_one<T, 1, 16, INT><<<dim3(bx, 1), 128, 0, s>>>(a);
    else k_one<T, 1, 8, INT><<<dim3(bx, 1), 128, 0, s>>>(a);
  } else if (a.F == 2) {
    k_one<T, 2, 8, INT><<<dim3(bx, 1), 128, 0, s>>>(a);
  } else {
    k_one<T, 4, 4, INT><<<dim3(bx, (unsigned)((a.F + 3) / 4)), 128, 0, s>>>(a);
  }
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}

static OneArgs one_args(const Plan *p, int F, float *cake, double *res) {
  OneArgs a{};
  a.g = p->one;
  a.terms = p->d_one_terms;
  a.cnt = p->d_one_cnt;
  a.slice_ptr = p->d_one_ptr;
  a.scale = p->d_one_scale;
  a.cake = cake;
  a.res = res;
  a.n_bins = p->n_bins;
  a.F = F;
  a.round_res = p->encoding == MI_ENC_CSR;
  a.tile_of_bin = p->d_one_tile;
  a.tiles = p->d_tiles;
  a.blobs = p->d_blobs;
  return a;
}

static int launch_one_chunk(Plan *p, const void *frames, int dtype, int F, int64_t stride, float *cake, double *partial,
                            bool want_lo, double *res, cudaStream_t s) {
  if (!want_lo) res = nullptr;
  else if (!res) res = p->one_res_in_xc ? (double *)p->d_xc : p->d_one_res;
  OneArgs a = one_args(p, F, cake, res);
  a.frames = frames;
  a.stride = stride;
  // without a dark its zeros are not read, except by a graph, which a later dark may follow
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if (!p->has_dark) MI_CUDA(cudaStreamIsCapturing(s, &cap));
  a.dark = cap == cudaStreamCaptureStatusNone ? nullptr : p->d_dark;
  int rc = MI_OK;
  if (p->encoding == MI_ENC_MMA) {
    rc = dtype == MI_DT_U8 ? launch_one_t<uint8_t, true>(p, a, s) : launch_one_t<uint16_t, true>(p, a, s);
  } else switch (dtype) {
    case MI_DT_U8: rc = launch_one_t<uint8_t, false>(p, a, s); break;
    case MI_DT_U16: rc = launch_one_t<uint16_t, false>(p, a, s); break;
    case MI_DT_U32: rc = launch_one_t<uint32_t, false>(p, a, s); break;
    case MI_DT_I64: rc = launch_one_t<int64_t, false>(p, a, s); break;
    case MI_DT_F32: rc = launch_one_t<float, false>(p, a, s); break;
    case MI_DT_F64: rc = launch_one_t<double, false>(p, a, s); break;
    case MI_DT_I32: rc = launch_one_t<int32_t, false>(p, a, s); break;
    default: return set_error(MI_E_ARG, "unknown dtype %d", dtype);
  }
  return rc || !want_lo ? rc : launch_one_partials(p, res, F, partial, s);
}

int launch_one(Plan *p, const void *frames, int dtype, int F, int64_t stride, float *cake, double *partial,
               bool want_lo, double *res, cudaStream_t s) {
  const size_t es = dtype_size(dtype);
  int rc = MI_OK;
  for (int f0 = 0; f0 < F && rc == MI_OK; f0 += kOneChunk)
    rc = launch_one_chunk(p, (const uint8_t *)frames + (size_t)f0 * stride * es, dtype, std::min(kOneChunk, F - f0),
                          stride, cake ? cake + (size_t)f0 * p->n_bins : nullptr,
                          partial + (size_t)f0 * p->n_r * p->n_slots * 2, want_lo, res, s);
  return rc;
}

// pixels of an eight-frame block: compact indices for panel plans, whose virtual detector is
// mostly outside the panels' spans, else the detector's
static int64_t pm_pixels(const Plan *p) { return p->panels.size() > 1 ? p->n_xc : (int64_t)p->ny * p->nz; }

// eight-frame blocks that fit the pixel-major buffer (256 B a referenced pixel) together with their bin
// results.  None where the referenced band is under an eighth of the detector and twice the bins (32 B a
// detector pixel for fp32), or the bins of a panel plan are over 3.5 a referenced pixel: over 16 wide
// frames then go through the fp32 rows and the run kernel
static int64_t pm_blocks(const Plan *p, bool want_lo) {
  const int64_t px = p->encoding == MI_ENC_MMA ? 2 : 4;   // bytes per pixel and frame
  const int64_t per = (pm_pixels(p) * px + (want_lo ? p->n_bins * 8 : 0)) * kPmFrames;
  return p->n_xc * kXcRowBytes / per;
}

bool one_pm_fits(const Plan *p, bool want_lo) {
  return (p->encoding == MI_ENC_RUNS || p->encoding == MI_ENC_MMA) && p->d_one_terms && p->n_xc > 0 &&
         pm_blocks(p, want_lo) >= 1;
}

// MMA plans of one detector
static int launch_one_pm16(Plan *p, const void *frames, int dtype, int F, int64_t stride, float *cake, double *partial,
                           bool want_lo, cudaStream_t s) {
  const int64_t n_px = pm_pixels(p);
  const int round = (int)std::min<int64_t>(pm_blocks(p, want_lo), kMaxFramesPerLaunch / kPmFrames) * kPmFrames;
  for (int f0 = 0; f0 < F; f0 += round) {
    const int nf = std::min(round, F - f0);
    const int nb = (nf + kPmFrames - 1) / kPmFrames;
    uint4 *pm = (uint4 *)p->d_xc;
    double *res = want_lo ? (double *)(pm + (int64_t)nb * n_px) : nullptr;
    const dim3 gs((unsigned)p->n_xchunks, (unsigned)nb);
    const void *src = (const uint8_t *)frames + (size_t)f0 * stride * dtype_size(dtype);
    if (dtype == MI_DT_U8) k_pm16<uint8_t><<<gs, 256, 0, s>>>((const uint8_t *)src, stride, nf, p->ny, p->d_xchunks, pm, n_px);
    else k_pm16<uint16_t><<<gs, 256, 0, s>>>((const uint16_t *)src, stride, nf, p->ny, p->d_xchunks, pm, n_px);
    MI_CUDA(cudaGetLastError());
    const OneArgs a = one_args(p, nf, cake ? cake + (size_t)f0 * p->n_bins : nullptr, res);
    const dim3 grid((unsigned)((p->one.n_slices * 32 + 127) / 128), (unsigned)nb);
    if (p->one.n_slices < kPlainDeep * (int64_t)std::max(p->n_sms, 1)) k_one_pm16<8><<<grid, 128, 0, s>>>(a, pm, n_px);
    else k_one_pm16<4><<<grid, 128, 0, s>>>(a, pm, n_px);
    MI_CUDA(cudaGetLastError());
    if (want_lo) {
      const int rc = launch_one_partials(p, res, nf, partial + (size_t)f0 * p->n_r * p->n_slots * 2, s);
      if (rc) return rc;
    }
  }
  return MI_OK;
}

template <typename T>
static void pm_launch(const Plan *p, const Plan::Panel &pn, const void *frames, int F, int64_t stride, float *pm,
                      cudaStream_t s) {
  const dim3 grid((unsigned)(pn.chunk_end - pn.chunk_begin), (unsigned)((F + kPmFrames - 1) / kPmFrames));
  if (grid.x == 0) return;
  k_pm<T><<<grid, 256, 0, s>>>((const T *)frames, stride, F, pn.ny, pn.z_off, p->ny, p->d_dark,
                               p->d_xchunks + pn.chunk_begin, pm, pm_pixels(p), p->panels.size() > 1);
}

int launch_one_pm(Plan *p, const void *const *frames, const int *dtypes, const int64_t *strides, int first, int F,
                  float *cake, double *partial, bool want_lo, cudaStream_t s) {
  if (p->encoding == MI_ENC_MMA) {
    const void *src = (const uint8_t *)frames[0] + (size_t)first * strides[0] * dtype_size(dtypes[0]);
    return launch_one_pm16(p, src, dtypes[0], F, strides[0], cake, partial, want_lo, s);
  }
  const int round = (int)std::min<int64_t>(pm_blocks(p, want_lo), kMaxFramesPerLaunch / kPmFrames) * kPmFrames;
  for (int f0 = 0; f0 < F; f0 += round) {
    const int nf = std::min(round, F - f0);
    const int nb = (nf + kPmFrames - 1) / kPmFrames;
    float *pm = (float *)p->d_xc;
    double *res = want_lo ? (double *)(pm + (int64_t)nb * pm_pixels(p) * kPmFrames) : nullptr;
    for (size_t i = 0; i < p->panels.size(); ++i) {
      const Plan::Panel &pn = p->panels[i];
      const void *src = (const uint8_t *)frames[i] + (size_t)(first + f0) * strides[i] * dtype_size(dtypes[i]);
      switch (dtypes[i]) {
        case MI_DT_U8: pm_launch<uint8_t>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_U16: pm_launch<uint16_t>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_U32: pm_launch<uint32_t>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_I64: pm_launch<int64_t>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_F32: pm_launch<float>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_F64: pm_launch<double>(p, pn, src, nf, strides[i], pm, s); break;
        case MI_DT_I32: pm_launch<int32_t>(p, pn, src, nf, strides[i], pm, s); break;
        default: return set_error(MI_E_ARG, "unknown dtype %d", dtypes[i]);
      }
      MI_CUDA(cudaGetLastError());
    }
    const OneArgs a = one_args(p, nf, cake ? cake + (size_t)f0 * p->n_bins : nullptr, res);
    const dim3 grid((unsigned)((p->one.n_slices * 32 + 127) / 128), (unsigned)nb);
    // terms in flight per lane as in the plain path's rule
    if (p->one.n_slices < kPlainDeep * (int64_t)std::max(p->n_sms, 1)) k_one_pm<8><<<grid, 128, 0, s>>>(a, pm, pm_pixels(p));
    else k_one_pm<4><<<grid, 128, 0, s>>>(a, pm, pm_pixels(p));
    MI_CUDA(cudaGetLastError());
    if (want_lo) {
      const int rc = launch_one_partials(p, res, nf, partial + (size_t)f0 * p->n_r * p->n_slots * 2, s);
      if (rc) return rc;
    }
  }
  return MI_OK;
}

}  // namespace mi
