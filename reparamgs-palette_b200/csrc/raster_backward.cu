// Tile compositing, adjoint (draw_weight_B / draw_color_B, gsplatcu/kernel.cu:
// 1176-1379).  The forward is in raster.cu.
//
// One 128-thread block per 16x16 tile; each of the 4 warps owns an 8x8 block
// and each lane two pixels of one column, four rows apart, so the
// per-Gaussian loop control and the warp reduction of the gradient terms are
// shared by 64 pixels.  Batches are staged and culled as in the forward: each
// record's mask of the quarters its cut ellipse can reach is found once, by
// the thread that stages it.  The warps walk their records from the last
// contributor to the front, two at a time: both records' opacity terms are
// evaluated before the two transmittance recoveries so that their exp()
// chains overlap, and the two records' gradient vectors are summed in one
// warp reduction.  Masks at staging and the exact skip threshold: 0.364 ->
// 0.329 ms at 1M Gaussians, 1080p (full adjoint, 500k: 0.609 -> 0.581 ms).
#include "gsb_geometry.cuh"
#include "gsb_internal.h"
#include "gsb_tiles.cuh"

namespace gsb {

constexpr int kBatch = 256;
constexpr int kAdjThreads = 128;  // two pixels per thread, 8x8 pixels per warp

struct PixelPair {
  int tx, ty;    // tile origin; the warp blocks are its 8x8 quarters
  int px;        // column
  int py0, py1;  // rows (py1 = py0 + 4)
};

__device__ __forceinline__ PixelPair pixels_of(int tile, int gx) {
  const int tx = tile % gx, ty = tile / gx;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  PixelPair p;
  p.tx = tx * kTile;
  p.ty = ty * kTile;
  p.px = p.tx + (w & 1) * 8 + (lane & 7);
  p.py0 = p.ty + (w >> 1) * 8 + (lane >> 3);
  p.py1 = p.py0 + 4;
  return p;
}

template <int K>
__device__ __forceinline__ void load_feats(const float4* srec, int j, float v2w, float* f) {
  f[0] = v2w;  // channel 0 sits in v1.w
#pragma unroll
  for (int k = 1; k < K; ++k) {
    const float4 q = srec[(2 + (k - 1) / 4) * kBatch + j];
    f[k] = ((k - 1) & 3) == 0 ? q.x : ((k - 1) & 3) == 1 ? q.y : ((k - 1) & 3) == 2 ? q.z : q.w;
  }
}

// Sum of NV per-lane values over groups of 2*OFF0 lanes (the whole warp for
// OFF0 = 16, each half-warp for OFF0 = 8) with NV-1 + log2(2*OFF0/NV)
// shuffles: each exchange step halves the values a lane carries (lanes with
// the step's bit set keep the upper half), so the totals end up spread over
// the group's lanes.  Returns this lane's total; *idx is the value index it
// holds and *owner is set on exactly one lane per index and group.
template <int NV, int OFF0 = 16>
__device__ __forceinline__ float warp_transpose_sum(float (&x)[NV], int lane, int* idx,
                                                    bool* owner) {
  static_assert(NV >= 1 && NV <= 2 * OFF0 && (NV & (NV - 1)) == 0,
                "NV must be a power of two no larger than the group");
  int id = 0;
  int off = OFF0;
#pragma unroll
  for (int w = NV / 2; w >= 1; w >>= 1, off >>= 1) {
    const bool hi = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float send = hi ? x[i] : x[i + w];
      const float keep = hi ? x[i + w] : x[i];
      x[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    id += hi ? w : 0;
  }
  float v = x[0];
#pragma unroll
  for (int o = off; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  *idx = id;
  *owner = off == 0 || (lane & (2 * off - 1)) == 0;  // NV == group size: every lane
  return v;
}

template <int NV>
struct Pow2 {
  static constexpr int value = NV <= 1 ? 1 : NV <= 2 ? 2 : NV <= 4 ? 4 : NV <= 8 ? 8 : NV <= 16 ? 16 : 32;
};

// Per-pixel back-to-front state of the adjoint.
template <int K>
struct BwdPixel {
  float dl[K], G[K];
  float T, Tf, dTf;
  int cont;
};

// One contributor of one pixel in the adjoint: recovers T, accumulates the
// pixel's gradient terms into x (x[0..K) features, then alpha, u, conic).
template <int K, bool GEOM, bool DTAU>
__device__ __forceinline__ bool adjoint_pixel(BwdPixel<K>& p, int idx, float m, float4 v0,
                                              float4 v1, float dx, float dy, const float4* srec,
                                              int jj, float* x) {
  if (!(idx < p.cont) || !(m >= v1.y)) return false;
  const float g = expf(m);
  const float ap = fminf(kAlphaMax, v1.z * g);
  const float one_m = 1.f - ap;
  p.T = __fdividef(p.T, one_m);
  const float wgt = ap * p.T;
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] += p.dl[k] * wgt;
  if (GEOM) {
    float f[K];
    load_feats<K>(srec, jj, v1.w, f);
    float dap = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      dap += p.dl[k] * (p.T * (f[k] - p.G[k]));
      p.G[k] = ap * f[k] + one_m * p.G[k];
    }
    if (DTAU) dap += p.dTf * __fdividef(-p.Tf, one_m);
    x[K] += dap * g;                                    // alpha
    x[K + 1] += dap * ((2.f * v0.z * dx + v0.w * dy) * ap);  // u.x
    x[K + 2] += dap * ((v0.w * dx + 2.f * v1.x * dy) * ap);  // u.y
    x[K + 3] += dap * (-0.5f * ap * (dx * dx));         // conic a
    x[K + 4] += dap * (-1.0f * ap * (dx * dy));         // conic b
    x[K + 5] += dap * (-0.5f * ap * (dy * dy));         // conic c
  }
  return true;
}

// Weights-only adjoint of two contributors at once: slot ja lies behind slot
// jb in list order, so it is undone first.  Both records' opacity terms are
// evaluated for both pixels before either transmittance update, so the four
// exp() chains overlap; the skip tests and the T recovery are exactly those
// of adjoint_pixel.  The two gradient vectors are summed together: one
// exchange at offset 16 leaves ja's partial sums on lanes 0-15 and jb's on
// lanes 16-31, then each half-warp transposes its K values (5 + 8 shuffles
// for K = 5, against 2 x 9 for two single reductions).  When at most
// kDirectLanes lanes hit each record, those lanes add their own sums
// directly (at most 2 x kDirectLanes x K atomics instead of about 60
// reduction instructions; 47 % of the records a warp visits have so few hits
// at 1M Gaussians, 1080p).  Measured, near / far view: 4 lanes 0.367 / 0.282
// ms, 8 lanes 0.362 / 0.278, 12 lanes 0.360 / 0.275, 16 lanes 0.361 / 0.278.
constexpr int kDirectLanes = 12;
template <int K>
__device__ __forceinline__ void adjoint_weights_pair(BwdPixel<K> (&p)[2], int base, int ja, int jb,
                                                     const float4* srec, const int32_t* sgid,
                                                     float fx, float fy0, float fy1, int lane,
                                                     float* __restrict__ dfeat) {
  const float4 a0 = srec[ja], a1 = srec[kBatch + ja];
  const float4 b0 = srec[jb], b1 = srec[kBatch + jb];
  const float fy[2] = {fy0, fy1};
  float apa[2], apb[2];
  bool ua[2], ub[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float dxa = a0.x - fx, dya = a0.y - fy[q];
    const float ma = fminf(0.f, half_form(a0.z, a0.w, a1.x, dxa, dya));
    apa[q] = fminf(kAlphaMax, a1.z * expf(ma));
    ua[q] = base + ja < p[q].cont && ma >= a1.y;
    const float dxb = b0.x - fx, dyb = b0.y - fy[q];
    const float mb = fminf(0.f, half_form(b0.z, b0.w, b1.x, dxb, dyb));
    apb[q] = fminf(kAlphaMax, b1.z * expf(mb));
    ub[q] = base + jb < p[q].cont && mb >= b1.y;
  }
  float xa[K], xb[K];
#pragma unroll
  for (int k = 0; k < K; ++k) xa[k] = xb[k] = 0.f;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (ua[q]) {
      p[q].T = __fdividef(p[q].T, 1.f - apa[q]);
      const float wgt = apa[q] * p[q].T;
#pragma unroll
      for (int k = 0; k < K; ++k) xa[k] += p[q].dl[k] * wgt;
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (ub[q]) {
      p[q].T = __fdividef(p[q].T, 1.f - apb[q]);
      const float wgt = apb[q] * p[q].T;
#pragma unroll
      for (int k = 0; k < K; ++k) xb[k] += p[q].dl[k] * wgt;
    }
  }
  const bool ha = ua[0] || ua[1], hb = ub[0] || ub[1];
  const unsigned ca = __ballot_sync(0xffffffffu, ha), cb = __ballot_sync(0xffffffffu, hb);
  if (!(ca | cb)) return;
  if (__popc(ca) <= kDirectLanes && __popc(cb) <= kDirectLanes) {
    if (ha) {
      const int64_t g = sgid[ja];
#pragma unroll
      for (int k = 0; k < K; ++k) atomicAdd(dfeat + g * K + k, xa[k]);
    }
    if (hb) {
      const int64_t g = sgid[jb];
#pragma unroll
      for (int k = 0; k < K; ++k) atomicAdd(dfeat + g * K + k, xb[k]);
    }
    return;
  }
  constexpr int NV = Pow2<K>::value;
  const bool hi = (lane & 16) != 0;
  float y[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (k < K) {
      const float send = hi ? xa[k] : xb[k];
      const float keep = hi ? xb[k] : xa[k];
      y[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    } else {
      y[k] = 0.f;
    }
  }
  int vidx;
  bool owner;
  const float tot = warp_transpose_sum<NV, 8>(y, lane, &vidx, &owner);
  if (owner && vidx < K && (hi ? cb : ca) != 0u) {
    const int64_t g = sgid[hi ? jb : ja];
    atomicAdd(dfeat + g * K + vidx, tot);
  }
}

// Destination of gradient value `v` of Gaussian g: x[0..K) features, then
// alpha, u (2), conic (3).
template <int K>
__device__ __forceinline__ float* grad_slot(int v, int64_t g, float* dfeat, float* dalpha,
                                            float* du, float* dconic) {
  if (v < K) return dfeat + g * K + v;
  if (v == K) return dalpha + g;
  if (v < K + 3) return du + 2 * g + (v - K - 1);
  return dconic + 3 * g + (v - K - 3);
}

// Full adjoint (GEOM) of two contributors at once, slot ja behind slot jb:
// the per-pixel terms are adjoint_pixel's, in the same order (ja then jb for
// each pixel).  The two gradient vectors (K + 6 values each) are summed
// together: one exchange at lane offset 16 leaves ja's partial sums on lanes
// 0-15 and jb's on lanes 16-31, then each half-warp transposes its values
// (K + 6 + 15 shuffles for the pair instead of 2 x 16 for K = 3..8).  When
// at most kDirectLanesGeom lanes hit each record, those lanes add their own
// K + 6 sums directly: at 1M / 1080p 0.776 -> 0.755 ms near, 0.462 -> 0.439
// ms far, against direct atomics for single hits only.
constexpr int kDirectLanesGeom = 8;
template <int K, bool DTAU>
__device__ __forceinline__ void adjoint_geom_pair(BwdPixel<K> (&p)[2], int base, int ja, int jb,
                                                  const float4* srec, const int32_t* sgid,
                                                  float fx, float fy0, float fy1, int lane,
                                                  float* __restrict__ dfeat,
                                                  float* __restrict__ dalpha,
                                                  float* __restrict__ du,
                                                  float* __restrict__ dconic) {
  constexpr int NREAL = K + 6;
  constexpr int NV = Pow2<NREAL>::value;
  static_assert(NV <= 16, "half-warp transposition holds at most 16 values");
  const float4 a0 = srec[ja], a1 = srec[kBatch + ja];
  const float4 b0 = srec[jb], b1 = srec[kBatch + jb];
  float xa[NV], xb[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) xa[v] = xb[v] = 0.f;
  const float dxa = a0.x - fx, dya0 = a0.y - fy0, dya1 = a0.y - fy1;
  const float dxb = b0.x - fx, dyb0 = b0.y - fy0, dyb1 = b0.y - fy1;
  const float ma0 = fminf(0.f, half_form(a0.z, a0.w, a1.x, dxa, dya0));
  const float ma1 = fminf(0.f, half_form(a0.z, a0.w, a1.x, dxa, dya1));
  const float mb0 = fminf(0.f, half_form(b0.z, b0.w, b1.x, dxb, dyb0));
  const float mb1 = fminf(0.f, half_form(b0.z, b0.w, b1.x, dxb, dyb1));
  bool ha = adjoint_pixel<K, true, DTAU>(p[0], base + ja, ma0, a0, a1, dxa, dya0, srec, ja, xa);
  bool hb = adjoint_pixel<K, true, DTAU>(p[0], base + jb, mb0, b0, b1, dxb, dyb0, srec, jb, xb);
  ha |= adjoint_pixel<K, true, DTAU>(p[1], base + ja, ma1, a0, a1, dxa, dya1, srec, ja, xa);
  hb |= adjoint_pixel<K, true, DTAU>(p[1], base + jb, mb1, b0, b1, dxb, dyb1, srec, jb, xb);
  const unsigned ca = __ballot_sync(0xffffffffu, ha), cb = __ballot_sync(0xffffffffu, hb);
  if (!(ca | cb)) return;
  if (__popc(ca) <= kDirectLanesGeom && __popc(cb) <= kDirectLanesGeom) {
    if (ha) {
      const int64_t g = sgid[ja];
#pragma unroll
      for (int v = 0; v < NREAL; ++v) atomicAdd(grad_slot<K>(v, g, dfeat, dalpha, du, dconic), xa[v]);
    }
    if (hb) {
      const int64_t g = sgid[jb];
#pragma unroll
      for (int v = 0; v < NREAL; ++v) atomicAdd(grad_slot<K>(v, g, dfeat, dalpha, du, dconic), xb[v]);
    }
    return;
  }
  const bool hi = (lane & 16) != 0;
  float y[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if (v < NREAL) {
      const float send = hi ? xa[v] : xb[v];
      const float keep = hi ? xb[v] : xa[v];
      y[v] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    } else {
      y[v] = 0.f;
    }
  }
  int vidx;
  bool owner;
  const float tot = warp_transpose_sum<NV, 8>(y, lane, &vidx, &owner);
  if (owner && vidx < NREAL && (hi ? cb : ca) != 0u) {
    const int64_t g = sgid[hi ? jb : ja];
    atomicAdd(grad_slot<K>(vidx, g, dfeat, dalpha, du, dconic), tot);
  }
}

// Walks each pixel's contributors back to front from its `contrib` index,
// recovering T by division by (1 - alpha') from the saved final T.  The
// per-pixel skip decisions use the forward's exact expressions, so the walk
// visits exactly the Gaussians the forward blended; T itself is recovered
// with a fast reciprocal division (relative error ~1e-7 per step).  Per
// Gaussian each lane first adds its two pixels' terms, then the warp's 64
// pixels are summed with one transposed reduction and added with one atomic
// per value.  GEOM adds the opacity / centre / conic adjoint (draw_color_B's
// terms, for any channel count); DTAU adds dL/dT_final
// (vanilla_3dgs/gsplatcu/kernel.cu:912-919).  As in the reference, the 0.99
// clamp and max(0, .) are not differentiated.  Weights-only, 8 blocks per SM
// (64 registers, a 12-byte spill): 0.377 -> 0.365 ms at 1M / 1080p against 7
// blocks (72 registers); the full adjoint 6 blocks per SM (80 registers):
// 0.755 -> 0.722 ms near, 1.146 -> 1.112 ms close, 0.437 -> 0.450 ms far.
template <int K, bool GEOM, bool DTAU>
__global__ void __launch_bounds__(kAdjThreads, GEOM ? 6 : 8)
    k_draw_backward(int H, int W, int gx, const int2* __restrict__ ranges,
                    const int32_t* __restrict__ gsid, const float4* __restrict__ records,
                    const int32_t* __restrict__ order,
                    const int32_t* __restrict__ contrib, const float* __restrict__ final_tau,
                    const float* __restrict__ dout, const float* __restrict__ dtau,
                    float* __restrict__ dfeat, float* __restrict__ dalpha,
                    float* __restrict__ du, float* __restrict__ dconic) {
  pdl_wait();
  constexpr int V = RecordLayout<K>::kVec4;
  constexpr int NREAL = GEOM ? K + 6 : K;
  constexpr int NV = Pow2<NREAL>::value;
  constexpr int kKeep = GEOM ? V - 1 : 2;  // float4s kept (v0, v1 and, with GEOM, the further channels)
  __shared__ float4 srec[kKeep * kBatch];
  __shared__ int32_t sgid[kBatch];
  __shared__ uint8_t smask[kBatch];
  __shared__ unsigned s_maxc;
  const int tile = order[blockIdx.x];
  const PixelPair pp = pixels_of(tile, gx);
  const int lane = threadIdx.x & 31;
  const int2 rg = ranges[tile];
  if (rg.y - rg.x == 0) return;  // uniform per block
  const int64_t hw = (int64_t)H * W;
  BwdPixel<K> p[2];
  const int rows[2] = {pp.py0, pp.py1};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const bool in = pp.px < W && rows[q] < H;
    const int64_t pix = (int64_t)rows[q] * W + pp.px;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      p[q].dl[k] = in ? dout[k * hw + pix] : 0.f;
      p[q].G[k] = 0.f;
    }
    p[q].Tf = in ? final_tau[pix] : 0.f;
    p[q].T = p[q].Tf;
    p[q].dTf = (DTAU && in) ? dtau[pix] : 0.f;
    p[q].cont = in ? contrib[pix] : 0;
  }
  const int wmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)max(p[0].cont, p[1].cont));
  if (threadIdx.x == 0) s_maxc = 0u;
  __syncthreads();
  if (lane == 0) atomicMax(&s_maxc, (unsigned)wmax);
  __syncthreads();
  // contributor indices never exceed the tile's list (clamped for safety
  // against mismatched inputs)
  const int maxc = min((int)s_maxc, rg.y - rg.x);
  const float fx = (float)pp.px, fy0 = (float)pp.py0, fy1 = (float)pp.py1;
  for (int top = maxc; top > 0; top -= kBatch) {
    const int base = max(0, top - kBatch);
    const int cnt = top - base;
    __syncthreads();
    for (int t = threadIdx.x; t < cnt; t += kAdjThreads) {
      const int g = gsid[rg.x + base + t];
      const float4* src = records + (int64_t)g * V;
      const float4 v0 = __ldg(src), v1 = __ldg(src + 1), v2 = __ldg(src + 2);
      srec[t] = v0;
      srec[kBatch + t] = v1;
#pragma unroll
      for (int v = 3; v < V; ++v)
        if (GEOM) srec[(v - 1) * kBatch + t] = __ldg(src + v);
      sgid[t] = g;
      smask[t] = (uint8_t)region_mask<2, 2, 8, 8>(v0, v1, v2, pp.tx, pp.ty);
    }
    __syncthreads();
    const int hi = min(cnt, wmax - base);
    for (int s_hi = hi; s_hi > 0; s_hi -= 32) {
      const int s_lo = max(0, s_hi - 32);
      const int j = s_lo + lane;
      unsigned mask = __ballot_sync(0xffffffffu, j < s_hi && ((smask[j] >> (threadIdx.x >> 5)) & 1));
      while (mask) {
        const int msb = 31 - __clz(mask);
        mask &= ~(1u << msb);
        if (mask) {
          const int msb2 = 31 - __clz(mask);
          mask &= ~(1u << msb2);
          if constexpr (GEOM)
            adjoint_geom_pair<K, DTAU>(p, base, s_lo + msb, s_lo + msb2, srec, sgid, fx, fy0, fy1,
                                       lane, dfeat, dalpha, du, dconic);
          else
            adjoint_weights_pair<K>(p, base, s_lo + msb, s_lo + msb2, srec, sgid, fx, fy0, fy1,
                                    lane, dfeat);
          continue;
        }
        const int jj = s_lo + msb;
        const int idx = base + jj;
        float x[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) x[v] = 0.f;
        const float4 v0 = srec[jj];
        const float4 v1 = srec[kBatch + jj];
        const float dx = v0.x - fx, dy0 = v0.y - fy0, dy1 = v0.y - fy1;
        const float m0 = fminf(0.f, half_form(v0.z, v0.w, v1.x, dx, dy0));
        const float m1 = fminf(0.f, half_form(v0.z, v0.w, v1.x, dx, dy1));
        bool hit = adjoint_pixel<K, GEOM, DTAU>(p[0], idx, m0, v0, v1, dx, dy0, srec, jj, x);
        hit |= adjoint_pixel<K, GEOM, DTAU>(p[1], idx, m1, v0, v1, dx, dy1, srec, jj, x);
        const unsigned cm = __ballot_sync(0xffffffffu, hit);
        if (!cm) continue;
        const int64_t g = sgid[jj];
        if (__popc(cm) == 1) {
          if (hit) {
#pragma unroll
            for (int k = 0; k < K; ++k) atomicAdd(dfeat + g * K + k, x[k]);
            if (GEOM) {
              atomicAdd(dalpha + g, x[K]);
              atomicAdd(du + 2 * g, x[K + 1]);
              atomicAdd(du + 2 * g + 1, x[K + 2]);
              atomicAdd(dconic + 3 * g, x[K + 3]);
              atomicAdd(dconic + 3 * g + 1, x[K + 4]);
              atomicAdd(dconic + 3 * g + 2, x[K + 5]);
            }
          }
          continue;
        }
        int vidx;
        bool owner;
        const float tot = warp_transpose_sum<NV>(x, lane, &vidx, &owner);
        if (owner && vidx < NREAL) {
          float* dst;
          if (vidx < K)
            dst = dfeat + g * K + vidx;
          else if (vidx == K)
            dst = dalpha + g;
          else if (vidx < K + 3)
            dst = du + 2 * g + (vidx - K - 1);
          else
            dst = dconic + 3 * g + (vidx - K - 3);
          atomicAdd(dst, tot);
        }
      }
    }
  }
}

template <int K>
static void draw_bwd_k(int tiles, int H, int W, int gx, const int2* rg, const int32_t* gsid,
                       const float4* rec, const int32_t* order, const int32_t* contrib,
                       const float* ft, const float* dout, const float* dtau, float* dfeat,
                       float* dalpha, float* du, float* dq, cudaStream_t st) {
  const bool geom = dalpha != nullptr;
  auto kern = (geom && dtau) ? k_draw_backward<K, true, true>
              : geom         ? k_draw_backward<K, true, false>
                             : k_draw_backward<K, false, false>;
  launch_pdl(kern, dim3(tiles), dim3(kAdjThreads), 0, st, H, W, gx, rg, gsid, rec, order, contrib,
             ft, dout, dtau, dfeat, dalpha, du, dq);
}

int launch_draw_backward(int64_t n, int H, int W, int channels, const int32_t* ranges,
                         const int32_t* gsid, const SplatState& s, const int32_t* contrib,
                         const float* final_tau, const float* dout, const float* dtau,
                         float* dfeat, float* dalpha, float* du, float* dconic, cudaStream_t st) {
  (void)n;
  const int gx = div_up(W, kTile), gy = div_up(H, kTile);
  const int tiles = gx * gy;
  if (tiles == 0) return GSB_OK;
  const int2* rg = (const int2*)ranges;
  if (channels < 1 || channels > 8) return GSB_ERR_INVALID_ARGUMENT;
  const int rc = launch_tile_order(rg, tiles, s.tile_order, st);
  if (rc) return rc;
  switch (channels) {
#define GSB_K(KK)                                                                              \
  case KK:                                                                                     \
    draw_bwd_k<KK>(tiles, H, W, gx, rg, gsid, s.records, s.tile_order, contrib, final_tau,      \
                   dout, dtau, dfeat, dalpha, du, dconic, st);                                 \
    break;
    GSB_K(1) GSB_K(2) GSB_K(3) GSB_K(4) GSB_K(5) GSB_K(6) GSB_K(7) GSB_K(8)
#undef GSB_K
    default: return GSB_ERR_INVALID_ARGUMENT;
  }
  return check_launch("splat_backward");
}

}  // namespace gsb
