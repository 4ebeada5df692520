// Culling shared by the compositing forward and its adjoint: which pixel
// blocks of a tile a record can reach.
#pragma once

#include "gsb_common.cuh"

namespace gsb {

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Which blocks of BW x BH pixels, of the region of NCOL x NROW blocks at pixel
// (X0, Y0), can the record's cut ellipse d^T Q d <= c2 reach?  Bit b * NCOL + c
// stands for column c of band b.  Evaluated once per record by the thread that
// stages it: every warp testing every record against its own block (support
// box, then the minimum of the form over the block's edges) took 10 % of the
// forward's instructions.  A clear bit only drops pixels whose quadratic form
// exceeds the cut (which is widened for the rounding of the FP32 form, see
// gsb_record.cuh), so the images do not depend on the mask.  Over a band the
// ellipse's right edge s dy + sqrt(A - B dy^2) is concave: its maximum is the
// support hx when the rightmost point lies in (or within a margin of) the
// band, else the value at one of the band's ends; the left edge likewise.
template <int NCOL, int NROW, int BW, int BH>
__device__ __forceinline__ unsigned region_mask(float4 v0, float4 v1, float4 v2, int X0, int Y0) {
  constexpr unsigned kAll = (1u << (NCOL * NROW)) - 1u;
  const float ux = v0.x, uy = v0.y, hx = v2.x, hy = v2.y, c2 = v2.z;
  const float qa = -2.f * v0.z, qb = -v0.w, qc = -2.f * v1.x;
  if (!(hx > -INFINITY)) return 0u;  // opacity below the threshold: blends nowhere
  if (!(c2 < INFINITY) || !isfinite(ux) || !isfinite(uy)) return kAll;  // unbounded
  const float ia = rcp_approx(qa), ic = rcp_approx(qc);
  const float s = -qb * ia, A = c2 * ia, B = (qa * qc - qb * qb) * ia * ia;
  const float dyr = -qb * ic * hx;  // the rightmost point's dy; the leftmost's is -dyr
  const float eps = 0.05f + 1e-3f * hy, xm = 0.02f + 1e-4f * hx;
  const float ox = ux - (float)X0, oy = (float)Y0 - uy;
  unsigned mask = 0u;
#pragma unroll
  for (int b = 0; b < NROW; ++b) {
    const float d1 = fmaxf(oy + (float)(BH * b), -hy);
    const float d2 = fminf(oy + (float)(BH * b + BH - 1), hy);
    if (d1 <= d2) {
      const float w1 = sqrt_approx(fmaxf(0.f, A - B * (d1 * d1)));
      const float w2 = sqrt_approx(fmaxf(0.f, A - B * (d2 * d2)));
      const float c1 = s * d1, c2b = s * d2;
      const bool rin = dyr >= d1 - eps && dyr <= d2 + eps;
      const bool lin = -dyr >= d1 - eps && -dyr <= d2 + eps;
      const float xr = rin ? hx : fmaxf(c1 + w1, c2b + w2) + xm;
      const float xl = lin ? -hx : fminf(c1 - w1, c2b - w2) - xm;
      const int lo = max(__float2int_ru(ox + xl), 0);
      const int hi = min(__float2int_rd(ox + xr), BW * NCOL - 1);
      if (lo <= hi) mask |= ((2u << (hi / BW)) - (1u << (lo / BW))) << (b * NCOL);
    }
  }
  return mask;
}

}  // namespace gsb
