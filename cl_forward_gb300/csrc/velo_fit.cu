// velo_fit.cu -- straight-line fit of every output track (x and y linear in
// z, least squares), the stage that follows the search in the pipeline the
// reference's input files come from (their track records carry a 4-float
// header; KernelDefinitions.h:25 defines the pixel weight PARAM_W, unused by
// the search).  Hits are weighted equally by PARAM_W = 3966.94 / mm^2, so the
// weight scales chi2 only.
//
// One CTA per event, one thread per track.  The sums and residuals are kept to
// 48 bits as unevaluated sums of two FP32 values (error-free transformations:
// Knuth's two-sum, and the product's rounding error by a fused multiply-add),
// of coordinates relative to the track's first hit, which is exact and takes
// the cancellation out of the sums; the 2 x 2 solution is in FP64.  The results
// are rounded to FP32 at the end, as those of an FP64 evaluation are, and lie
// as near to the exact ones.
//
// GB300 issues an FP64 instruction of a warp every 16 cycles per SM, an FP32
// one every quarter cycle: the FP64 sums, residuals and divisions (some 350 a
// track) bounded the kernel: 1.49 ms for 1.54 M tracks of 10,000 events, now
// 0.38 ms.  Root-mean-square error against extended precision 2.5e-8 of the
// values before and after, the rounding to FP32.
#include <cuda_runtime.h>

#include "velo_internal.h"

namespace velo {
namespace {

constexpr double kPixelWeight = 3966.94;   // PARAM_W, KernelDefinitions.h:25
constexpr int kFitThreads = 64;

// The fit in FP64 throughout, for tracks whose coordinates leave the range in
// which the FP32 pairs are exact.
__device__ __noinline__ velo_track_fit fit_fp64(const velo_track& tr, uint32_t n, int H, const float* x,
                                                const float* y, const float* z) {
  double s0 = 0, sz = 0, szz = 0, sx = 0, sxz = 0, sy = 0, syz = 0;
  for (uint32_t k = 0; k < n; ++k) {
    const uint32_t h = tr.hits[k];
    if (h >= (uint32_t)H) continue;
    const double zz = z[h], xx = x[h], yy = y[h];
    s0 += 1;
    sz += zz;
    szz += zz * zz;
    sx += xx;
    sxz += xx * zz;
    sy += yy;
    syz += yy * zz;
  }
  velo_track_fit out{0.f, 0.f, 0.f, 0.f, 0.f};
  const double det = s0 * szz - sz * sz;
  if (s0 >= 2 && det > 0) {
    const double tx = (s0 * sxz - sz * sx) / det, ty = (s0 * syz - sz * sy) / det;
    const double x0 = (sx - tx * sz) / s0, y0 = (sy - ty * sz) / s0;
    double chi2 = 0;
    for (uint32_t k = 0; k < n; ++k) {
      const uint32_t h = tr.hits[k];
      if (h >= (uint32_t)H) continue;
      const double rx = x[h] - (x0 + tx * z[h]), ry = y[h] - (y0 + ty * z[h]);
      chi2 += kPixelWeight * (rx * rx + ry * ry);
    }
    const double ndf = 2.0 * s0 - 4.0;
    out.x0 = (float)x0;
    out.tx = (float)tx;
    out.y0 = (float)y0;
    out.ty = (float)ty;
    out.chi2_ndf = ndf > 0 ? (float)(chi2 / ndf) : 0.f;
  }
  return out;
}

// h + l, |l| at most half an ulp of h.
struct Pair {
  float h, l;
};

__device__ __forceinline__ Pair two_sum(float a, float b) {   // exact
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return Pair{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ Pair difference(float a, float b) { return two_sum(a, -b); }
__device__ __forceinline__ Pair renormalised(float h, float l) {
  const float s = __fadd_rn(h, l);
  return Pair{s, __fsub_rn(l, __fsub_rn(s, h))};
}
__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
  const Pair s = two_sum(a.h, b.h);
  return renormalised(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ Pair operator-(Pair a) { return Pair{-a.h, -a.l}; }
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
  const float p = __fmul_rn(a.h, b.h);
  return Pair{p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p)))};
}
__device__ __forceinline__ Pair pair_of(double v) {
  const float h = (float)v;
  return Pair{h, (float)(v - (double)h)};
}
__device__ __forceinline__ double value(Pair a) { return (double)a.h + (double)a.l; }

// A difference of two coordinates with which products and their rounding
// errors stay in FP32's normal range.
__device__ __forceinline__ bool in_range(Pair d) {
  const float a = fabsf(d.h);
  return a < 1e6f && (a > 1e-9f || a == 0.f);
}

__global__ void __launch_bounds__(kFitThreads) fit_tracks_kernel(const uint8_t* input, const uint64_t* ev_offset,
                                                                 const uint32_t* ev_valid, const velo_track* tracks,
                                                                 const uint32_t* counts, const uint64_t* first,
                                                                 int n_events, velo_track_fit* fits) {
  const int e = blockIdx.x;
  if (e >= n_events || !ev_valid[e]) return;
  const int32_t* hdr = reinterpret_cast<const int32_t*>(input + ev_offset[e]);
  const int S = hdr[0], H = hdr[1];
  const float* x = reinterpret_cast<const float*>(hdr + 2 + 3 * S + H);
  const float* y = x + H;
  const float* z = y + H;
  const uint64_t f0 = first[e];
  for (uint32_t t = threadIdx.x; t < counts[e]; t += blockDim.x) {
    const velo_track& tr = tracks[f0 + t];
    const uint32_t n = tr.hitsNum < VELO_MAX_TRACK_SIZE ? tr.hitsNum : VELO_MAX_TRACK_SIZE;
    // sums of u = z - z of the first hit, v = x - ..., w = y - ...
    float x1 = 0.f, y1 = 0.f, z1 = 0.f;
    int hits = 0;
    bool ok = true;
    const Pair zero{0.f, 0.f};
    Pair su = zero, suu = zero, sv = zero, svu = zero, sw = zero, swu = zero;
    for (uint32_t k = 0; k < n; ++k) {
      const uint32_t h = tr.hits[k];
      if (h >= (uint32_t)H) continue;
      const float hx = x[h], hy = y[h], hz = z[h];
      if (hits++ == 0) {   // contributes nothing relative to itself
        x1 = hx;
        y1 = hy;
        z1 = hz;
        continue;
      }
      const Pair u = difference(hz, z1), v = difference(hx, x1), w = difference(hy, y1);
      ok = ok && in_range(u) && in_range(v) && in_range(w);
      su = su + u;
      suu = suu + u * u;
      sv = sv + v;
      svu = svu + v * u;
      sw = sw + w;
      swu = swu + w * u;
    }
    ok = ok && fmaxf(fabsf(x1), fmaxf(fabsf(y1), fabsf(z1))) < 1e6f;
    velo_track_fit out{0.f, 0.f, 0.f, 0.f, 0.f};
    if (!ok) {
      out = fit_fp64(tr, n, H, x, y, z);
    } else if (hits >= 2) {
      const double s0 = hits, du = value(su), dv = value(sv), dw = value(sw);
      const double det = s0 * value(suu) - du * du;
      if (det > 0) {
        const double inv = 1.0 / det, inv0 = 1.0 / s0;
        const double tx = (s0 * value(svu) - du * dv) * inv, ty = (s0 * value(swu) - du * dw) * inv;
        const double a = (dv - tx * du) * inv0, b = (dw - ty * du) * inv0;   // the line at z1, relative to x1 and y1
        const Pair ptx = pair_of(-tx), pty = pair_of(-ty), pa = pair_of(-a), pb = pair_of(-b);
        Pair chi2 = zero;
        for (uint32_t k = 0; k < n; ++k) {
          const uint32_t h = tr.hits[k];
          if (h >= (uint32_t)H) continue;
          const Pair u = difference(z[h], z1);
          const Pair rx = (difference(x[h], x1) + ptx * u) + pa, ry = (difference(y[h], y1) + pty * u) + pb;
          chi2 = chi2 + (rx * rx + ry * ry);
        }
        out.x0 = (float)(x1 + (a - tx * z1));
        out.tx = (float)tx;
        out.y0 = (float)(y1 + (b - ty * z1));
        out.ty = (float)ty;
        out.chi2_ndf = hits > 2 ? (float)(kPixelWeight * value(chi2) * (0.5 / (s0 - 2.0))) : 0.f;
      }
    }
    fits[f0 + t] = out;
  }
}

}  // namespace

int launch_fit_tracks(const uint8_t* input, const uint64_t* ev_offset, const uint32_t* ev_valid,
                      const velo_track* tracks, const uint32_t* counts, const uint64_t* first, int n_events,
                      velo_track_fit* fits, void* stream) {
  if (n_events <= 0) return 0;
  fit_tracks_kernel<<<n_events, kFitThreads, 0, (cudaStream_t)stream>>>(input, ev_offset, ev_valid, tracks, counts, first,
                                                                n_events, fits);
  return (int)cudaGetLastError();
}

}  // namespace velo
