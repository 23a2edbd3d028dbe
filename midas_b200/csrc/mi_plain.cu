// mi_plain.cu -- kernel (a) (cast + dark, 128-bit vector loads) and the plain
// one-frame-per-launch path that runs the reference's own GPU algorithm:
//   process_direct_kernel<T>             FF_HEDM/src/IntegratorFitPeaksGPUStream.cu:1148-1160
//   integrate_noMapMask                  IntegratorFitPeaksGPUStream.cu:975-1050
//     (one thread per bin, FP32 accumulation in record order, bilinear resampling at
//      FP32 positions in gradient mode, FP64 cake)
//   calculate_1D_profile_kernel          IntegratorFitPeaksGPUStream.cu:1162-1254
//   calculate_1D_profile_simple_mean_kernel  IntegratorFitPeaksGPUStream.cu:1256-1334
// The plain path is the baseline the batched kernel is measured against; it is
// written here from the algorithm, not copied.
#include <stdint.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "mi_internal.h"

namespace mi {

// ---------------------------------------------------------------------------
// kernel (a): out[f][p] = (float)in[f][p] - dark[p], 16-byte loads of the input
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float cvt(T v) {
  return (float)v;
}

template <typename T>
__global__ void k_cast_vec(const T *__restrict__ in, int64_t n_pixels, int n_frames,
                           const float *__restrict__ dark, float *__restrict__ out) {
  constexpr int V = 16 / sizeof(T);  // elements per 128-bit load
  const int64_t nvec = n_pixels / V;
  const int64_t total = nvec * n_frames;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = i / nvec, v = i - f * nvec;
    const int64_t p0 = v * V;
    union {
      uint4 u;
      T e[V];
    } x;
    x.u = __ldg((const uint4 *)(in + f * n_pixels) + v);
    float r[V];
#pragma unroll
    for (int k = 0; k < V; ++k) r[k] = cvt(x.e[k]);
    if (dark) {
      if (V >= 4) {
#pragma unroll
        for (int k = 0; k < V; k += 4) {
          const float4 d = __ldg((const float4 *)(dark + p0 + k));
          r[k] -= d.x; r[k + 1] -= d.y; r[k + 2] -= d.z; r[k + 3] -= d.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k) r[k] -= __ldg(dark + p0 + k);
      }
    }
    float *o = out + f * n_pixels + p0;
    if (V >= 4 && (n_pixels % 4) == 0) {
#pragma unroll
      for (int k = 0; k < V; k += 4) *(float4 *)(o + k) = make_float4(r[k], r[k + 1], r[k + 2], r[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) o[k] = r[k];
    }
  }
}

template <typename T>
__global__ void k_cast_scalar(const T *__restrict__ in, int64_t n_pixels, int n_frames, int64_t start,
                              const float *__restrict__ dark, float *__restrict__ out) {
  const int64_t per = n_pixels - start;
  const int64_t total = per * n_frames;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = i / per, p = start + (i - f * per);
    float r = cvt(in[f * n_pixels + p]);
    if (dark) r -= dark[p];
    out[f * n_pixels + p] = r;
  }
}

static int grid_for(int64_t work, int threads) {
  int64_t g = (work + threads - 1) / threads;
  const int64_t cap = 148 * 16;  // persistent-style cap: 16 CTAs per SM on 148 SMs
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

template <typename T>
static int cast_t(const void *frames, int64_t n_pixels, int n_frames, const float *dark, float *out,
                  cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const T *in = (const T *)frames;
  const bool aligned = ((uintptr_t)in % 16 == 0) && ((uintptr_t)out % 16 == 0) &&
                       (!dark || (uintptr_t)dark % 16 == 0) && (n_pixels % V == 0);
  int64_t start = 0;
  if (aligned) {
    const int64_t work = (n_pixels / V) * n_frames;
    k_cast_vec<T><<<grid_for(work, 256), 256, 0, s>>>(in, n_pixels, n_frames, dark, out);
    MI_CUDA(cudaGetLastError());
    start = n_pixels;
  }
  if (start < n_pixels) {
    k_cast_scalar<T><<<grid_for((n_pixels - start) * n_frames, 256), 256, 0, s>>>(in, n_pixels, n_frames,
                                                                                start, dark, out);
    MI_CUDA(cudaGetLastError());
  }
  return MI_OK;
}

int launch_cast(const void *frames, int dtype, int64_t n_pixels, int n_frames, const float *dark, float *out,
                cudaStream_t s) {
  switch (dtype) {
    case MI_DT_U8: return cast_t<uint8_t>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_U16: return cast_t<uint16_t>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_U32: return cast_t<uint32_t>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_I64: return cast_t<int64_t>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_F32: return cast_t<float>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_F64: return cast_t<double>(frames, n_pixels, n_frames, dark, out, s);
    case MI_DT_I32: return cast_t<int32_t>(frames, n_pixels, n_frames, dark, out, s);
  }
  return set_error(MI_E_ARG, "unknown dtype %d", dtype);
}

// ---------------------------------------------------------------------------
// plain integration: one thread per bin, the reference's FP32 sum over the bin's records in
// their order.
//
// Layout: 32 bins (a block of 8 R rows x 4 eta columns, so a warp's pixels are neighbours) form
// a slice; step k of a slice holds record k of each bin that has one, packed side by side, so a
// warp's loads are contiguous and nothing is padded: a lane's place is its rank among the lanes
// still active.  A record is what its sum needs and no more: {pixel, frac} in floor mode (8 B),
// {base pixel, y and z fraction, frac} otherwise (16 B): the resampled position depends on the
// map alone and is worked out once, when the plan is made (k_plain_fill).
// Bounded by the latency of the gathers at few bins and by L1 gathers at many (2048^2, 1980 x 180
// gradient: L1 80 % busy, DRAM 49).  Thread per bin
// over bin-major records (20 B, resampled in every call) took 378 us for the 2048^2, 1980 x 180
// gradient map, 147 us for 1024^2, 495 x 45 floor and 482 us for 2880^2, 3960 x 360 gradient
// (21 M records); this takes 52, 21 and 97 us (cold caches; the last 3.7 TB/s), same bits.  Blocks
// of 4 x 8 bins measured 58 / 77 / 102 us, rows of 32 columns 97 / 81 / 147 (before the records
// were fetched ahead: 52 / 79 / 90).
// ---------------------------------------------------------------------------
__global__ void k_plain_count(PlainLayout g, const int32_t *nmap, int32_t *cnt, int64_t *slice_n) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= g.n_slices) return;
  const int64_t b = plain_bin(g, s, lane);
  const int n = b >= 0 ? nmap[2 * b] : 0;
  cnt[s * 32 + lane] = n;
  int64_t t = n;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) slice_n[s] = t;
}

__global__ void k_plain_fill(PlainLayout g, PlainFill f) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= g.n_slices) return;
  const int64_t b = plain_bin(g, s, lane);
  const int n = f.cnt[s * 32 + lane];
  const int64_t j0 = b >= 0 ? f.nmap[2 * b + 1] : 0;
  int64_t at = f.slice_ptr[s];
  float A = 0.0f;
  for (int k = 0; __any_sync(0xffffffffu, k < n); ++k) {
    const int64_t o = plain_step(k < n, lane, at);
    if (k >= n) continue;
    const mi_map_record r = f.recs[j0 + k];
    const float w = (float)r.frac;
    A += r.areaWeight;
    if (f.mode == MI_MODE_FLOOR) {
      // PrecomputeOffsets_kernel: the flat index evaluated in float (GPU stream), or the
      // truncated pixel where it lies on the detector (midas_integrate)
      const long long ty = (long long)r.y, tz = (long long)r.z;
      long long o2 = (long long)((float)(tz * (long long)f.ny) + r.y);
      if (f.sem == MI_SEM_PY) o2 = ty >= 0 && ty < f.ny && tz >= 0 && tz < f.nz ? tz * f.ny + ty : -1;
      else if (o2 < 0 || o2 >= (long long)f.ny * f.nz) o2 = -1;
      f.t2[o] = make_uint2((uint32_t)(int)o2, __float_as_uint(w));
    } else {
      float ry = r.y, rz = r.z;
      if (f.mode == MI_MODE_GRADIENT) {
        const float dy = ry - f.bc_y, dz = rz - f.bc_z;
        const float R = sqrtf(dy * dy + dz * dz);
        if (R > 1.0f) {
          const float d = r.deltaR;
          ry -= d * dy / R;
          rz -= d * dz / R;
        }
      }
      int iy = (int)floorf(ry), iz = (int)floorf(rz);
      float fy = ry - (float)iy, fz = rz - (float)iz;
      if (iy < 0) { iy = 0; fy = 0.0f; }
      if (iy >= f.ny - 1) { iy = f.ny - 2; fy = 1.0f; }
      if (iz < 0) { iz = 0; fz = 0.0f; }
      if (iz >= f.nz - 1) { iz = f.nz - 2; fz = 1.0f; }
      f.t4[o] = make_uint4((uint32_t)(iz * f.ny + iy), __float_as_uint(fy), __float_as_uint(fz), __float_as_uint(w));
    }
  }
  if (b >= 0) f.area_gs[b] = A;
}

struct PlainArgs {
  PlainLayout g;
  const uint2 *t2;
  const uint4 *t4;
  const int32_t *cnt;
  const int64_t *slice_ptr;
  const double *area_in;
  const float *area_gs;
  const float *img;
  double *cake;
  int ny, sem, normalize;
};

// U: records whose pixels a lane has in flight, with as many records fetched ahead
template <bool FLOOR, int U>
__global__ void __launch_bounds__(128) k_plain_integrate(PlainArgs a) {
  using R = typename std::conditional<FLOOR, uint2, uint4>::type;
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.g.n_slices) return;
  const int64_t s = a.g.n_slices - 1 - i;   // outer rings hold more records: they start first
  const int64_t b = plain_bin(a.g, s, lane);
  const int n = a.cnt[s * 32 + lane];
  int n_max = n;
  for (int o = 16; o > 0; o >>= 1) n_max = max(n_max, __shfl_xor_sync(0xffffffffu, n_max, o));
  const int64_t first = a.slice_ptr[s];
  int64_t at = first;
  const R *tab = FLOOR ? (const R *)a.t2 : (const R *)a.t4;
  float I = 0.0f;
  R t[U];
  if (n_max > 0) plain_load<R, U>(tab, first, 0, n, lane, at, t);
  for (int k = 0; k < n_max; k += U) {
    R tn[U];
    if (k + U < n_max) plain_load<R, U>(tab, first, k + U, n, lane, at, tn);
    if constexpr (FLOOR) {
      float v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldg(a.img + max((int)t[u].x, 0));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float In = I + ((int)t[u].x >= 0 ? v[u] : 0.0f) * __uint_as_float(t[u].y);
        I = k + u < n ? In : I;
      }
    } else {
      float c[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float *p = a.img + (int)t[u].x;
        c[u][0] = __ldg(p); c[u][1] = __ldg(p + 1); c[u][2] = __ldg(p + a.ny); c[u][3] = __ldg(p + a.ny + 1);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float fy = __uint_as_float(t[u].y), fz = __uint_as_float(t[u].z);
        const float v = c[u][0] * (1.0f - fy) * (1.0f - fz) + c[u][1] * fy * (1.0f - fz) +
                        c[u][2] * (1.0f - fy) * fz + c[u][3] * fy * fz;
        const float In = I + v * __uint_as_float(t[u].w);
        I = k + u < n ? In : I;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = tn[u];
  }
  if (b < 0) return;
  double out;
  if (a.sem == MI_SEM_GPUSTREAM) {
    const float A = a.area_gs[b];
    out = (A > (float)kAreaThreshold) ? (a.normalize ? (double)(I / A) : (double)I) : 0.0;
  } else {
    const double ai = a.area_in[b];
    out = a.normalize ? (ai > kAreaThreshold ? (double)I / ai : 0.0) : (double)I;
  }
  a.cake[b] = out;
}

// The one-frame path's records, laid out on the device from the map's.  On a stream of its own
// with stream-ordered scratch: a plan made while a server runs must not wait for the device.
int build_plain(Plan *p, const mi_map_record *recs, const int32_t *nmap, size_t *acct) {
  p->plain = plain_layout(p->n_r, p->n_eta);
  const PlainLayout &g = p->plain;
  const int64_t n_pix = (int64_t)p->ny * p->nz;
  cudaStream_t st = nullptr;
  MI_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  std::vector<void *> tmp;
  auto temp = [&](void **q, size_t bytes) {
    cudaError_t e = cudaMallocAsync(q, std::max<size_t>(bytes, 16), st);
    if (e == cudaSuccess) tmp.push_back(*q);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
  };
  auto keep = [&](void **q, size_t bytes) {
    *acct += std::max<size_t>(bytes, 16);
    return cudaMalloc(q, std::max<size_t>(bytes, 16));
  };
  auto build = [&]() -> int {
    int32_t *d_nmap = nullptr;
    int64_t *d_n = nullptr;
    mi_map_record *d_recs = nullptr;
    // the map on the device while its layout is made: in the pixel-major buffer, which is large
    // enough for most maps and not in use yet, else in scratch
    const size_t b_recs = sizeof(mi_map_record) * p->n_records, b_n = sizeof(int64_t) * g.n_slices;
    const size_t b_nmap = sizeof(int32_t) * 2 * p->n_bins, need = b_recs + b_n + b_nmap;
    uint8_t *at = p->d_xc;
    if (!at || (size_t)p->n_xc * kXcRowBytes < need) MI_CUDA(temp((void **)&at, need));
    d_recs = (mi_map_record *)at;
    d_n = (int64_t *)(at + b_recs);
    d_nmap = (int32_t *)(at + b_recs + b_n);
    MI_CUDA(copy_pieces(d_nmap, nmap, b_nmap, cudaMemcpyHostToDevice));
    if (p->n_records > 0) MI_CUDA(copy_pieces(d_recs, recs, b_recs, cudaMemcpyHostToDevice));
    MI_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // a pageable copy's last piece may still be under way
    MI_CUDA(keep((void **)&p->d_plain_cnt, sizeof(int32_t) * 32 * g.n_slices));
    MI_CUDA(keep((void **)&p->d_plain_ptr, sizeof(int64_t) * g.n_slices));
    MI_CUDA(keep((void **)&p->d_area_gs, sizeof(float) * p->n_bins));
    const unsigned blocks = (unsigned)((g.n_slices * 32 + 127) / 128);
    k_plain_count<<<blocks, 128, 0, st>>>(g, d_nmap, p->d_plain_cnt, d_n);
    MI_CUDA(cudaGetLastError());
    std::vector<int64_t> n(g.n_slices);
    MI_CUDA(cudaMemcpyAsync(n.data(), d_n, sizeof(int64_t) * g.n_slices, cudaMemcpyDeviceToHost, st));
    MI_CUDA(cudaStreamSynchronize(st));
    int64_t total = 0;
    for (int64_t &v : n) {
      const int64_t c = v;
      v = total;
      total += c;
    }
    MI_CUDA(cudaMemcpyAsync(p->d_plain_ptr, n.data(), sizeof(int64_t) * g.n_slices, cudaMemcpyHostToDevice, st));
    if (p->mode == MI_MODE_FLOOR) MI_CUDA(keep((void **)&p->d_plain_t2, sizeof(uint2) * total));
    else MI_CUDA(keep((void **)&p->d_plain_t4, sizeof(uint4) * total));
    PlainFill f{d_recs, d_nmap, p->d_plain_cnt, p->d_plain_ptr, p->d_plain_t2, p->d_plain_t4, p->d_area_gs,
                p->ny, p->nz, p->mode, p->semantics, (float)p->bc_y, (float)p->bc_z};
    k_plain_fill<<<blocks, 128, 0, st>>>(g, f);
    MI_CUDA(cudaGetLastError());
    MI_CUDA(cudaStreamSynchronize(st));
    MI_CUDA(cudaMalloc((void **)&p->d_plain_img, n_pix * sizeof(float)));
    *acct += n_pix * sizeof(float);
    return MI_OK;
  };
  const int rc = build();
  for (void *q : tmp) cudaFreeAsync(q, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return rc;
}

// one block per (R row, frame); both profiles in one pass.  variance != 0: the cake holds
// bin variances and the profiles are propagated variances (profile_1d_with_variance,
// packages/midas_integrate/midas_integrate/kernels.py:604-645): sum(A^2 V) / (sum A)^2 and
// sum(V) / N^2
template <typename T>
__global__ void k_profile(const T *cake, const double *area_in, int n_r, int n_eta, double *lo_aw,
                          double *lo_sm, int variance, int omp) {
  const int r = blockIdx.x;
  const int64_t f = blockIdx.y;
  if (r >= n_r) return;
  const T *ck = cake + f * (int64_t)n_r * n_eta;
  double s_ia = 0.0, s_a = 0.0, s_i = 0.0;
  int n = 0;
  for (int e = threadIdx.x; e < n_eta; e += blockDim.x) {
    const int64_t b = (int64_t)r * n_eta + e;
    const double A = area_in[b];
    const double I = (double)ck[b];
    if (omp) {
      // IntegratorZarrOMP.c:1829-1843: the mean of the row's nonzero, non-NaN bins; the
      // area-weighted mean over its valid, non-NaN bins
      if (!isnan(I)) {
        if (A > kAreaThreshold) {
          s_ia += I * A;
          s_a += A;
        }
        if (I != 0.0) {
          s_i += I;
          ++n;
        }
      }
    } else if (A > kAreaThreshold) {
      s_ia += variance ? I * A * A : I * A;
      s_a += A;
      s_i += I;
      ++n;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s_ia += __shfl_down_sync(0xffffffffu, s_ia, o);
    s_a += __shfl_down_sync(0xffffffffu, s_a, o);
    s_i += __shfl_down_sync(0xffffffffu, s_i, o);
    n += __shfl_down_sync(0xffffffffu, n, o);
  }
  __shared__ double sh[4][32];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    sh[0][wid] = s_ia; sh[1][wid] = s_a; sh[2][wid] = s_i; sh[3][wid] = (double)n;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t_ia = 0, t_a = 0, t_i = 0, t_n = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      t_ia += sh[0][k]; t_a += sh[1][k]; t_i += sh[2][k]; t_n += sh[3][k];
    }
    const double d_a = variance ? t_a * t_a : t_a, d_n = variance ? t_n * t_n : t_n;
    if (lo_aw) lo_aw[f * n_r + r] = t_a > kAreaThreshold ? t_ia / d_a : 0.0;
    if (lo_sm) lo_sm[f * n_r + r] = t_n > 0 ? t_i / d_n : 0.0;
  }
}

int launch_profile(Plan *p, const void *cake, int cake_dtype, int n_frames, double *lo_aw, double *lo_sm,
                   cudaStream_t s) {
  if (n_frames <= 0 || (!lo_aw && !lo_sm)) return MI_OK;
  if (n_frames > 65535) return set_error(MI_E_RANGE, "mi_profile_batch: more than 65535 frames per call");
  const dim3 grid((unsigned)p->n_r, (unsigned)n_frames);
  if (cake_dtype == MI_DT_F32)
    k_profile<float><<<grid, 256, 0, s>>>((const float *)cake, p->d_area_in, p->n_r, p->n_eta, lo_aw, lo_sm,
                                          p->variance, p->semantics == MI_SEM_OMP);
  else if (cake_dtype == MI_DT_F64)
    k_profile<double><<<grid, 256, 0, s>>>((const double *)cake, p->d_area_in, p->n_r, p->n_eta, lo_aw, lo_sm,
                                           p->variance, p->semantics == MI_SEM_OMP);
  else
    return set_error(MI_E_ARG, "mi_profile_batch: cake dtype must be MI_DT_F32 or MI_DT_F64");
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}

__global__ void k_nan_bins(float *cake, int64_t n_bins, const int32_t *bins, int n, int F) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)n * F) return;
  const int64_t f = i / n;
  cake[f * n_bins + bins[i % n]] = __int_as_float(0x7fc00000);
}

int launch_nan_bins(Plan *p, float *cake, int n_frames, cudaStream_t s) {
  if (!cake || p->n_nan_bins == 0 || n_frames <= 0) return MI_OK;
  const int64_t n = (int64_t)p->n_nan_bins * n_frames;
  k_nan_bins<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cake, p->n_bins, p->d_nan_bins, p->n_nan_bins, n_frames);
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}

// SumImages (IntegratorFitPeaksGPUStream.cu:1043-1046 into dSumMatrix, allocated at
// :2141-2144): sum[b] += cake[f][b] over the batch's frames, in FP64, frames in order (the
// reference adds per frame with atomics in any order); NaN bins (masked bins of the OpenMP
// semantics) add nothing.  Thread per bin; eight frames' loads in flight before the adds.
__global__ void k_sum_cake(const float *__restrict__ cake, int F, int64_t n_bins, double *__restrict__ sum) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < n_bins; b += step) {
    double s = sum[b];
    int f = 0;
    for (; f + 8 <= F; f += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldcs(cake + (int64_t)(f + u) * n_bins + b);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += isnan(v[u]) ? 0.0 : (double)v[u];
    }
    for (; f < F; ++f) {
      const float v = __ldcs(cake + (int64_t)f * n_bins + b);
      s += isnan(v) ? 0.0 : (double)v;
    }
    sum[b] = s;
  }
}

int launch_sum_cake(Plan *p, const float *cake, int n_frames, double *sum, cudaStream_t s) {
  if (n_frames <= 0 || p->n_bins == 0) return MI_OK;
  const int64_t blocks = std::min<int64_t>((p->n_bins + 255) / 256, (int64_t)std::max(p->n_sms, 1) * 8);
  k_sum_cake<<<(unsigned)blocks, 256, 0, s>>>(cake, n_frames, p->n_bins, sum);
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}

int launch_plain(Plan *p, const void *frame, int dtype, double *cake, double *lo_aw, double *lo_sm,
                 cudaStream_t s) {
  if (!cake) return set_error(MI_E_ARG, "mi_integrate_plain: cake output is required");
  const int64_t n_pix = (int64_t)p->ny * p->nz;
  int rc = launch_cast(frame, dtype, n_pix, 1, p->has_dark ? p->d_dark : nullptr, p->d_plain_img, s);
  if (rc) return rc;
  PlainArgs a;
  a.g = p->plain;
  a.t2 = p->d_plain_t2;
  a.t4 = p->d_plain_t4;
  a.cnt = p->d_plain_cnt;
  a.slice_ptr = p->d_plain_ptr;
  a.area_in = p->d_area_in;
  a.area_gs = p->d_area_gs;
  a.img = p->d_plain_img;
  a.cake = cake;
  a.ny = p->ny;
  a.sem = p->semantics;
  a.normalize = p->normalize;
  const unsigned blocks = (unsigned)((p->plain.n_slices * 32 + 127) / 128);
  // maps of few bins leave the chip to a few warps: more records in flight per lane; maps of many
  // bins (few records each) hide the latency with warps and lose by the registers.  Deep against
  // shallow, us: 744 slices 21 / 36 (floor), 2230 slices 28 / 45 (floor), 58 / 91 (gradient), 5580
  // slices 21.8 / 22.6, 11,160 slices 33 / 27 (floor), 59 / 52 (gradient), 44,550 slices 69 / 53,
  // 113 / 97
  const bool deep = p->plain.n_slices < kPlainDeep * (int64_t)std::max(p->n_sms, 1);
  if (p->mode == MI_MODE_FLOOR) {
    if (deep) k_plain_integrate<true, 16><<<blocks, 128, 0, s>>>(a);
    else k_plain_integrate<true, 8><<<blocks, 128, 0, s>>>(a);
  } else {
    if (deep) k_plain_integrate<false, 8><<<blocks, 128, 0, s>>>(a);
    else k_plain_integrate<false, 4><<<blocks, 128, 0, s>>>(a);
  }
  MI_CUDA(cudaGetLastError());
  return launch_profile(p, cake, MI_DT_F64, 1, lo_aw, lo_sm, s);
}

}  // namespace mi
