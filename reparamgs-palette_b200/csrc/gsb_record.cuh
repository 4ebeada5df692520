// The packed compositing record of one Gaussian (one per Gaussian, gathered
// per patch by the compositing kernels), as float4s:
//   v0  ux uy a b            centre; a = -qa / 2, b = -qb (conic qa, qb, qc)
//   v1  c p* alpha ch0       c = -qc / 2, skip threshold, opacity, channel 0
//   v2  hx hy c2 0           support half-extents and cut, for the culling
//   v3  ch1 ch2 ch3 ch4 ...  further channels (weights / colours), zero padded
// (record_channel(k) is the float index of channel k; RecordLayout<K>).
//
// With the conic scaled by -1/2 (exact), half_form gives p = -m / 2 of the
// Mahalanobis form m bit for bit, the argument of exp(): alpha' = min(0.99,
// alpha exp(min(p, 0))).  The reference skips a pixel whose alpha' is below
// 0.002 (gsplatcu/kernel.cu:343-353).  expf is non-decreasing over [-104, 0],
// and so is the rounded product with alpha, so the pixels it skips are exactly
// those with p < p*, the smallest p that is not skipped: one comparison
// decides, and the exponential is needed only for its value.
// tests/test_gpu_skip_threshold.py compares both float by float, around the
// thresholds and over runs of consecutive floats, and allows no mismatch: run it
// after a change of toolkit or of the math flags.  Outside of this are inputs that
// no covariance and no sigmoid gives: conics above 1e37, whose m overflows at another
// pixel than p, and an opacity of -infinity, which the reference blends as 0.99
// where exp() underflows (-inf * 0 is NaN) and which never blends here.
//
// Pixels outside the support box u +- (hx, hy) satisfy d^T Q d > c2, and any
// pixel with d^T Q d > c2 is skipped: c2 = 2 ln(alpha/0.002) + margin, widened
// for the rounding error of the FP32 quadratic form (proportional to the
// conic's condition number).  Degenerate or non-finite conics get an unbounded
// box and c2 = +inf (never culled); alpha < 0.002 an empty box (never blends).
#pragma once

#include "gsb_common.cuh"

namespace gsb {

// Does the reference blend a pixel with this p (<= 0)?
__device__ __forceinline__ bool record_blends(float a, float p) {
  return !(fminf(kAlphaMax, a * expf(p)) < kAlphaMin);
}

// p*: the smallest p <= 0 that blends, +1 if none does, -inf if all do.  The
// search gallops from the analytic value ln(0.002 / a), whose rounding leaves
// it a few floats away, then bisects; every loop ends because the candidates'
// bit patterns are bounded.
__device__ __forceinline__ float skip_threshold(float a) {
  if (!record_blends(a, 0.f)) return 1.f;
  if (record_blends(a, -INFINITY)) return -INFINITY;
  const uint32_t kInf = 0x7f800000u;  // bits of |p|: blends at 0, not at kInf
  const auto blends = [a](uint32_t bits) { return record_blends(a, -__uint_as_float(bits)); };
  const float guess = fabsf(fminf(0.f, logf(kAlphaMin / a)));
  uint32_t lo = min(__float_as_uint(guess), kInf - 1), hi, step = 1;
  if (blends(lo)) {
    hi = lo + 1;
    while (hi < kInf && blends(hi)) {
      lo = hi;
      step *= 2;
      hi = kInf - lo > step ? lo + step : kInf;
    }
  } else {
    hi = lo;
    lo = hi - 1;
    while (lo > 0 && !blends(lo)) {
      hi = lo;
      step *= 2;
      lo = hi > step ? hi - step : 0;
    }
  }
  while (hi - lo > 1) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (blends(mid))
      lo = mid;
    else
      hi = mid;
  }
  return -__uint_as_float(lo);
}

// Fills the record's geometry floats and zeroes the channel slots (the
// caller writes the channels at record_channel(k)).
__device__ __forceinline__ void record_head(float ux, float uy, float qa, float qb, float qc,
                                            float a, float* f) {
  const float cut = 2.f * logf(a / kAlphaMin) + kCutMargin;
  float hx = INFINITY, hy = INFINITY, c2 = INFINITY;
  if (cut < 0.f) {  // alpha < 0.002: never blends, empty box
    hx = hy = -INFINITY;
    c2 = cut;
  } else if (isfinite(cut) && isfinite(ux) && isfinite(uy)) {
    const float det = qa * qc - qb * qb;
    const float kappa = (qa + qc) * (qa + qc) / det;
    if (det > 0.f && qa > 0.f && qc > 0.f && kappa < 1e5f) {
      const float cw = cut * (1.f + 4e-6f * kappa) + 1e-3f;
      const float ex = sqrtf(cw * qc / det) * 1.0001f + 0.02f;
      const float ey = sqrtf(cw * qa / det) * 1.0001f + 0.02f;
      if (isfinite(ex) && isfinite(ey)) {
        hx = ex;
        hy = ey;
        c2 = cw;
      }
    }
  }
#pragma unroll
  for (int k = 12; k < 20; ++k) f[k] = 0.f;
  f[0] = ux;
  f[1] = uy;
  f[2] = -0.5f * qa;
  f[3] = -qb;
  f[4] = -0.5f * qc;
  f[5] = skip_threshold(a);
  f[6] = a;
  f[7] = 0.f;
  f[8] = hx;
  f[9] = hy;
  f[10] = c2;
  f[11] = 0.f;
}

}  // namespace gsb
