// mi_fit.cu -- kernel (d): batched Levenberg-Marquardt pseudo-Voigt peak fits.
//
// One warp per one to eight (frame, peak) windows of the eta-averaged lineouts.  Window
// selection and initial guesses follow fitPeaks / pf_estimate_initial_params
// (FF_HEDM/src/PeakFit.c:218-250, 275-470): nearest bin to the requested peak
// position (rejected unless closer than 2 bins), ROI of +-half_window bins,
// background guess from the ROI ends, amplitude above background, FWHM from a
// half-maximum walk.  The reference minimises the same least-squares objective
// with NLopt L-BFGS; here it is minimised with Levenberg-Marquardt: residuals,
// Jacobian and model in FP32 on lane-strided samples, the normal equations
// J^T J and J^T r reduced across the warp in FP64 and solved by an FP64
// Cholesky factorisation (one lane per window).  The centre
// is carried relative to the window centre so FP32 keeps sub-1e-5 px
// resolution; the final centre and 2-theta are formed in FP64.
//
// Models
//   MI_FIT_PV : b0 + b1*xn + h*(eta*L + (1-eta)*G), L = 1/(1+u^2),
//               G = exp(-ln2*u^2), u = (x-c)/(w/2)           params c,h,w,eta,b0,b1
//   MI_FIT_TCH: area-normalised Thompson-Cox-Hastings pseudo-Voigt + 2-term
//               Chebyshev background (pf_calculate_model, PeakFit.c:50-92;
//               FWHM/eta from sig, gam per pf_tch_eta_fwhm, PeakFit.c:17-42)
//                                                             params A,c,sig,gam,b0,b1
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "mi_fitcore.cuh"
#include "mi_internal.h"

namespace mi {

constexpr int kNP = 6;
constexpr int kNTri = kNP * (kNP + 1) / 2;  // lower triangle of J^T J
constexpr int kNSum = kNTri + kNP + 1;      // sums of one evaluation: J^T J, J^T r, chi^2
constexpr int kMaxWin = 1024;  // samples per window (lane-strided)
constexpr int kFitWarps = 4;   // warps per block

struct FitArgs {
  const double *x, *lo, *peaks;
  int F, n_x, n_peaks, half, max_iter, slots, model;
  double x_bin, px, lsd;
  double *out;
  int32_t *iters;
};

// model value and gradient at local x (relative to the window centre), xn in [-1, 1]
__device__ inline float model(int kind, const float *p, float xl, float xn, float *g) {
  if (kind == MI_FIT_PV) {
    const float c = p[0], h = p[1], w = fmaxf(p[2], 1e-6f), et = p[3];
    const float hw = 0.5f * w;
    const float u = (xl - c) / hw, u2 = u * u;
    const float L = 1.0f / (1.0f + u2);
    const float G = expf(-0.69314718f * u2);
    const float P = et * L + (1.0f - et) * G;
    const float dP_du2 = -et * L * L - (1.0f - et) * 0.69314718f * G;
    g[0] = h * dP_du2 * (-2.0f * u / hw);
    g[1] = P;
    g[2] = h * dP_du2 * (-u2 / hw);
    g[3] = h * (L - G);
    g[4] = 1.0f;
    g[5] = xn;
    return p[4] + p[5] * xn + h * P;
  }
  // TCH, area normalised
  const float A = p[0], c = p[1];
  float F, et, dF_ds, dF_dg, de_ds, de_dg;
  tch(p[2], p[3], &F, &et, &dF_ds, &dF_dg, &de_ds, &de_dg);
  const float sg = F * 0.42466090014400953f;  // FWHM / (2 sqrt(2 ln 2))
  const float Gn = 0.3989422804014327f / sg;  // 1 / (sg sqrt(2 pi))
  const float hw = 0.5f * F;
  const float dx = xl - c, dx2 = dx * dx;
  const float eg = expf(-0.5f * dx2 / (sg * sg));
  const float G = Gn * eg;
  const float den = dx2 + hw * hw;
  const float L = 0.3183098861837907f * hw / den;  // (hw/pi) / (dx^2 + hw^2)
  const float P = et * L + (1.0f - et) * G;
  // derivatives w.r.t. centre and FWHM
  const float dG_dc = G * dx / (sg * sg);
  const float dL_dc = L * 2.0f * dx / den;
  const float dsg_dF = 0.42466090014400953f;
  const float dG_dsg = G * (-1.0f / sg + dx2 / (sg * sg * sg));
  const float dL_dhw = 0.3183098861837907f * (den - 2.0f * hw * hw) / (den * den);
  const float dP_dF = et * dL_dhw * 0.5f + (1.0f - et) * dG_dsg * dsg_dF;
  const float dP_de = L - G;
  g[0] = P;
  g[1] = A * (et * dL_dc + (1.0f - et) * dG_dc);
  g[2] = A * (dP_dF * dF_ds + dP_de * de_ds);
  g[3] = A * (dP_dF * dF_dg + dP_de * de_dg);
  g[4] = 1.0f;
  g[5] = xn;
  return p[4] + p[5] * xn + A * P;
}

// Solve (J^T J + lam diag) d = J^T r by Cholesky, unrolled into registers: nrm holds the lower
// triangle of J^T J row by row, then J^T r.
__device__ __forceinline__ bool chol_solve(const double *nrm, double lam, double *x) {
  double L[kNTri];
  bool ok = true;
#pragma unroll
  for (int i = 0; i < kNP; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      const double a = nrm[i * (i + 1) / 2 + j];
      double s = i == j ? a + lam * fmax(a, 1e-30) : a;
#pragma unroll
      for (int k = 0; k < j; ++k) s -= L[i * (i + 1) / 2 + k] * L[j * (j + 1) / 2 + k];
      if (i == j) {
        ok = ok && s > 0.0;
        L[i * (i + 1) / 2 + i] = sqrt(s);
      } else {
        L[i * (i + 1) / 2 + j] = s / L[j * (j + 1) / 2 + j];
      }
    }
  double y[kNP];
#pragma unroll
  for (int i = 0; i < kNP; ++i) {
    double s = nrm[kNTri + i];
#pragma unroll
    for (int k = 0; k < i; ++k) s -= L[i * (i + 1) / 2 + k] * y[k];
    y[i] = s / L[i * (i + 1) / 2 + i];
  }
#pragma unroll
  for (int i = kNP - 1; i >= 0; --i) {
    double s = y[i];
#pragma unroll
    for (int k = i + 1; k < kNP; ++k) s -= L[k * (k + 1) / 2 + i] * x[k];
    x[i] = s / L[i * (i + 1) / 2 + i];
  }
  return ok;
}

__device__ inline void clamp_params(int kind, float *p, float half_span, float x_bin) {
  if (kind == MI_FIT_PV) {
    p[0] = fminf(fmaxf(p[0], -half_span), half_span);
    p[1] = fmaxf(p[1], 0.0f);
    p[2] = fminf(fmaxf(p[2], 0.05f * x_bin), 4.0f * half_span);
    p[3] = fminf(fmaxf(p[3], 0.0f), 1.0f);
  } else {
    p[0] = fmaxf(p[0], 0.0f);
    p[1] = fminf(fmaxf(p[1], -half_span), half_span);
    p[2] = fmaxf(p[2], 1e-6f);
    p[3] = fmaxf(p[3], 0.01f);
  }
}

// Shared memory of one window slot: two sets of normal sums (the accepted parameters' and the
// trial's), the trial parameters (16-byte aligned; 6 floats and a double), the samples y, xl, xn.
__host__ __device__ inline uint32_t fit_slot_bytes(int n_cap) {
  return (uint32_t)(2 * 8 * kNSum + 4 * 8 + 16 * n_cap + 15) & ~15u;
}

// One warp fits `slots` consecutive windows in lockstep.  Per iteration lane w solves window
// w's damped normal equations and decides on its step (the serial FP64 chain runs for all the
// warp's windows at once), and the whole warp evaluates one window after another, lane =
// sample.
//   PV: an evaluation's sums serve an accepted step as they are, one evaluation an iteration.
//   TCH: an accepted step is evaluated again.  The compiler contracts the two evaluations of
//   the TCH derivatives differently in their last bits, and the ill-conditioned (sig, gam)
//   pair turns a last bit into another path of the iteration; evaluating both keeps the
//   results of a fit what they always were.
// What bounds it: instruction issue and the fixed latencies of the serial solve at 21 % of the warps
// (14,080 windows: issue slots 56 % busy, FP64 pipe 27, memory idle), and for a few windows the solve's
// chain alone.  A solve by every
// lane of a warp for its one window, all-reduced sums and two evaluations took 2.68 ms for
// 14,080 PV windows of 31 samples; this takes 0.37 ms, and 80 us where it
// took 160 for the 10 windows of one lineout (same bits).
template <int KIND>
__global__ void __launch_bounds__(32 * kFitWarps, 4) k_fit(FitArgs a) {
  extern __shared__ __align__(16) uint8_t fsm[];
  const int kind = KIND == MI_FIT_PV ? MI_FIT_PV : a.model;
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5, W = a.slots;
  const int64_t total = (int64_t)a.F * a.n_peaks;
  const int64_t w0 = ((int64_t)blockIdx.x * kFitWarps + wl) * W;
  if (w0 >= total) return;
  const int n_win = (int)min((int64_t)W, total - w0);
  const int n_cap = 2 * a.half + 1;
  const uint32_t sb = fit_slot_bytes(n_cap);
  uint8_t *base = fsm + (size_t)wl * W * sb;
  auto slot_sum = [&](int w, int buf) { return (double *)(base + (size_t)w * sb) + buf * kNSum; };
  auto slot_pn = [&](int w) { return (float *)(slot_sum(w, 2)); };
  auto slot_trial = [&](int w) { return slot_sum(w, 2) + 3; };   // TCH: chi^2 of the trial
  auto slot_y = [&](int w) { return slot_sum(w, 2) + 4; };
  auto slot_xl = [&](int w) { return (float *)(slot_y(w) + n_cap); };
  auto slot_xn = [&](int w) { return slot_xl(w) + n_cap; };

  // ---- windows: nearest bin, samples; lane w keeps what window w needs
  int my_n = 0, my_at = 0, my_it = 0;
  double my_xref = 0.0;
  float my_span = 0.0f;
  for (int w = 0; w < n_win; ++w) {
    const int64_t wid = w0 + w;
    const int f = (int)(wid / a.n_peaks), pk = (int)(wid % a.n_peaks);
    const double *x = a.x;
    const double *y = a.lo + (int64_t)f * a.n_x;
    const double loc = a.peaks[pk];
    int best = -1;
    double bd = 1e300;
#pragma unroll 4
    for (int i = lane; i < a.n_x; i += 32) {
      const double d = fabs(x[i] - loc);
      if (d < bd || (d == bd && i < best)) { bd = d; best = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double od = __shfl_xor_sync(0xffffffffu, bd, o);
      const int ob = __shfl_xor_sync(0xffffffffu, best, o);
      if (od < bd || (od == bd && ob < best)) { bd = od; best = ob; }
    }
    int n = 0, why = -1;
    if (best >= 0 && bd < 2.0 * a.x_bin) {
      const int s0 = max(0, best - a.half), s1 = min(a.n_x - 1, best + a.half);
      n = s1 - s0 + 1;
      if (n < kNP + 1 || n > kMaxWin) { n = 0; why = -2; }
      if (n > 0) {
        const double xref = x[best];
        const double xlo = x[s0], xhi = x[s1];
        const double xr = fmax(xhi - xlo, 1e-12);
        for (int i = lane; i < n; i += 32) {
          const double xi = x[s0 + i];
          slot_y(w)[i] = y[s0 + i];
          slot_xl(w)[i] = (float)(xi - xref);
          slot_xn(w)[i] = (float)(2.0 * (xi - xlo) / xr - 1.0);
        }
        if (lane == w) {
          my_n = n;
          my_at = best - s0;
          my_xref = xref;
          my_span = (float)fmax(xhi - xref, xref - xlo);
        }
      }
    }
    if (n == 0) {
      if (lane < MI_FIT_NOUT) a.out[wid * MI_FIT_NOUT + lane] = 0.0;
      if (lane == 0) a.iters[wid] = why;
    }
  }
  __syncwarp();

  // ---- initial guess (pf_estimate_initial_params), lane w for window w
  float p[kNP], pn[kNP];
#pragma unroll
  for (int u = 0; u < kNP; ++u) p[u] = pn[u] = 0.0f;
  if (my_n > 0) {
    const double *y = slot_y(lane);
    const int n = my_n;
    const int bgw = max(1, min(5, n / 4));
    double bgs = 0.0;
    for (int i = 0; i < bgw; ++i) bgs += y[i] + y[n - 1 - i];
    const double bg = bgs / (2.0 * bgw);
    double amp = y[my_at] - bg;
    if (amp <= 0) amp = y[my_at];
    const double hm = bg + 0.5 * amp;
    int li = my_at, ri = my_at;
    while (li > 0 && y[li] > hm) --li;
    while (ri < n - 1 && y[ri] > hm) ++ri;
    double fwb = (double)(ri - li);
    if (!(fwb > 1.0)) fwb = 2.0;
    const double fwx = fwb * a.x_bin;
    if (KIND == MI_FIT_PV) {
      p[0] = 0.0f; p[1] = (float)amp; p[2] = (float)fwx; p[3] = 0.5f; p[4] = (float)bg; p[5] = 0.0f;
    } else {
      const double fg0 = 0.5 * fwx;
      double sg = (fg0 * 100.0) * (fg0 * 100.0) / 5.545177444479562;
      if (sg < 1e-6) sg = 1.0;
      double gm = fwx * 0.5 * 100.0;
      if (gm < 0.01) gm = 1.0;
      double ar = amp * fwx * 1.5;
      if (ar <= 0) ar = 1.0;
      p[0] = (float)ar; p[1] = 0.0f; p[2] = (float)sg; p[3] = (float)gm; p[4] = (float)bg; p[5] = 0.0f;
    }
    clamp_params(KIND, p, my_span, (float)a.x_bin);
  }

  // ---- LM.  first: the sums at the initial parameters are taken as they are
  double lam = 1e-3, chi2 = 0.0;
  int cur = 0, stall = 0;
  bool live = my_n > 0, first = true;
  for (;;) {
    // lane w: the trial of window w
    bool want = live;
    if (live) {
      if (first) {
#pragma unroll
        for (int u = 0; u < kNP; ++u) pn[u] = p[u];
      } else {
        double nrm[kNTri + kNP], d[kNP];
        const double *src = slot_sum(lane, cur);
#pragma unroll
        for (int q = 0; q < kNTri + kNP; ++q) nrm[q] = src[q];
        want = chol_solve(nrm, lam, d);
#pragma unroll
        for (int u = 0; u < kNP; ++u) pn[u] = (float)((double)p[u] + d[u]);
        clamp_params(KIND, pn, my_span, (float)a.x_bin);
      }
      float *q = slot_pn(lane);
      *(float4 *)q = make_float4(pn[0], pn[1], pn[2], pn[3]);
      *(float2 *)(q + 4) = make_float2(pn[4], pn[5]);
    }
    const uint32_t todo = __ballot_sync(0xffffffffu, want);
    __syncwarp();
    for (uint32_t t = todo; t; t &= t - 1) {
      const int w = __ffs(t) - 1;
      const int n = __shfl_sync(0xffffffffu, my_n, w);
      const int buf = __shfl_sync(0xffffffffu, cur, w) ^ 1;
      float pp[kNP];
      const float *q = slot_pn(w);
      const float4 q4 = *(const float4 *)q;
      const float2 q2 = *(const float2 *)(q + 4);
      pp[0] = q4.x; pp[1] = q4.y; pp[2] = q4.z; pp[3] = q4.w; pp[4] = q2.x; pp[5] = q2.y;
      const double *y = slot_y(w);
      const float *xl = slot_xl(w), *xn = slot_xn(w);
      auto eval = [&]() {
        double acc[kNSum];
#pragma unroll
        for (int k = 0; k < kNSum; ++k) acc[k] = 0.0;
        for (int i = lane; i < n; i += 32) {
          float g[kNP];
          const float m = model(kind, pp, xl[i], xn[i], g);
          const float r = (float)(y[i] - (double)m);
          int z = 0;
#pragma unroll
          for (int u = 0; u < kNP; ++u)
#pragma unroll
            for (int v = 0; v <= u; ++v) acc[z++] += (double)g[u] * (double)g[v];
#pragma unroll
          for (int u = 0; u < kNP; ++u) acc[z++] += (double)g[u] * (double)r;
          acc[z] += (double)r * (double)r;
        }
        return warp_sums<kNSum>(acc, lane);
      };
      double s = eval();
      if (KIND != MI_FIT_PV && !first) {
        const double c2n = __shfl_sync(0xffffffffu, s, kNSum - 1);
        const double c2 = __shfl_sync(0xffffffffu, chi2, w);
        if (lane == 0) *slot_trial(w) = c2n;
        if (c2n <= c2) s = eval();
      }
      if (lane < kNSum) slot_sum(w, buf)[lane] = s;
    }
    __syncwarp();
    // lane w: accept or reject
    if (live) {
      if (first) {
        cur ^= 1;
        chi2 = slot_sum(lane, cur)[kNSum - 1];
        live = a.max_iter > 0;
      } else {
        const double c2a = want ? slot_sum(lane, cur ^ 1)[kNSum - 1] : 0.0;
        const double c2n = KIND == MI_FIT_PV ? c2a : *slot_trial(lane);
        ++my_it;
        if (want && c2n <= chi2) {
          double rel = 0.0;
#pragma unroll
          for (int u = 0; u < kNP; ++u)
            rel = fmax(rel, fabs((double)pn[u] - (double)p[u]) / fmax(fabs((double)p[u]), 1e-3));
          const double dec = chi2 - c2n;
#pragma unroll
          for (int u = 0; u < kNP; ++u) p[u] = pn[u];
          cur ^= 1;
          chi2 = c2a;
          lam = fmax(lam * 0.1, 1e-12);
          if (rel < 1e-6 || dec <= 1e-9 * chi2) {
            if (++stall >= 2) live = false;
          } else {
            stall = 0;
          }
        } else {
          lam *= 10.0;
          if (lam > 1e12) live = false;
        }
        if (my_it >= a.max_iter) live = false;
      }
    }
    first = false;
    if (!__any_sync(0xffffffffu, live)) break;
    __syncwarp();
  }
  // ---- outputs (FP64): [area, center, sig, gam, fwhm, eta, chi2_dof, height, bg0, bg1, 2theta]
  if (my_n > 0) {
    double *out = a.out + (w0 + lane) * MI_FIT_NOUT;
    double area, center, sig, gam, fw, et, height;
    if (KIND == MI_FIT_PV) {
      center = my_xref + (double)p[0];
      height = p[1];
      fw = p[2];
      et = p[3];
      area = height * fw * (et * 1.5707963267948966 + (1.0 - et) * 1.0644670194312262);
      sig = 0.0;
      gam = 0.0;
    } else {
      float F, e2, t0, t1, t2, t3;
      tch(p[2], p[3], &F, &e2, &t0, &t1, &t2, &t3);
      area = p[0];
      center = my_xref + (double)p[1];
      sig = p[2];
      gam = p[3];
      fw = F;
      et = e2;
      const double sgm = fw * 0.42466090014400953;
      height = area * (et * (2.0 / (3.141592653589793 * fw)) + (1.0 - et) * 0.3989422804014327 / sgm);
    }
    out[0] = area;
    out[1] = center;
    out[2] = sig;
    out[3] = gam;
    out[4] = fw;
    out[5] = et;
    out[6] = chi2 / fmax((double)(my_n - kNP), 1.0);
    out[7] = height;
    out[8] = p[4];
    out[9] = p[5];
    out[10] = (a.px > 0 && a.lsd > 0) ? atan(center * a.px / a.lsd) * 57.29577951308232 : 0.0;
    a.iters[w0 + lane] = my_it;
  }
}

}  // namespace mi

using namespace mi;

extern "C" int mi_fit_batch(const double *x, const double *lineouts, int n_frames, int n_x, const double *peaks,
                            int n_peaks, const mi_fit_opts *opts, double *out, int32_t *iters, void *stream) {
  if (!x || !lineouts || !peaks || !opts || !out || !iters) return set_error(MI_E_ARG, "mi_fit_batch: null argument");
  if (n_frames < 0 || n_x < 0 || n_peaks < 0) return set_error(MI_E_ARG, "mi_fit_batch: negative size");
  if (opts->model != MI_FIT_PV && opts->model != MI_FIT_TCH)
    return set_error(MI_E_ARG, "mi_fit_batch: unknown model %d", opts->model);
  if (opts->half_window < 3 || 2 * opts->half_window + 1 > kMaxWin)
    return set_error(MI_E_RANGE, "mi_fit_batch: half_window must be in [3, %d]", (kMaxWin - 1) / 2);
  if (!(opts->x_bin > 0)) return set_error(MI_E_ARG, "mi_fit_batch: x_bin must be > 0");
  if (n_frames == 0 || n_peaks == 0 || n_x == 0) return MI_OK;
  FitArgs a;
  a.x = x;
  a.lo = lineouts;
  a.peaks = peaks;
  a.F = n_frames;
  a.n_x = n_x;
  a.n_peaks = n_peaks;
  a.half = opts->half_window;
  a.max_iter = opts->max_iter > 0 ? opts->max_iter : 100;
  a.x_bin = opts->x_bin;
  a.px = opts->px_um;
  a.lsd = opts->lsd_um;
  a.out = out;
  a.iters = iters;
  const int64_t windows = (int64_t)n_frames * n_peaks;
  // windows per warp: one while they cannot fill the device (the shortest chain per window),
  // then as many as keep every window of the call resident at once, up to 8 (14,080 windows:
  // 469 us with at most 4, 373 with 8, 372 with 16; 50,000: 1365, 1147, 1151)
  const uint32_t sb = fit_slot_bytes(2 * a.half + 1);
  int dev = 0, sms = 0, dev_smem = 0;
  MI_CUDA(cudaGetDevice(&dev));
  MI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MI_CUDA(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const int64_t warps = (int64_t)sms * kFitWarps * 4;
  const int64_t fit = std::max<int64_t>(1, (48 * 1024 / kFitWarps) / sb);
  a.slots = (int)std::min<int64_t>(std::min<int64_t>(8, fit), (windows + warps - 1) / warps);
  const int64_t per_block = (int64_t)kFitWarps * a.slots;
  const int64_t blocks = (windows + per_block - 1) / per_block;
  if (blocks > INT32_MAX) return set_error(MI_E_RANGE, "mi_fit_batch: too many windows");
  const uint32_t smem = kFitWarps * (uint32_t)a.slots * sb;
  a.model = opts->model;
  auto kern = opts->model == MI_FIT_PV ? k_fit<MI_FIT_PV> : k_fit<MI_FIT_TCH>;
  if (smem > 48 * 1024) MI_CUDA(allow_smem(kern, dev_smem));
  kern<<<(unsigned)blocks, 32 * kFitWarps, smem, (cudaStream_t)stream>>>(a);
  MI_CUDA(cudaGetLastError());
  return MI_OK;
}
