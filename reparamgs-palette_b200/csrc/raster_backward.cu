// Tile compositing, adjoint (draw_weight_B / draw_color_B, gsplatcu/kernel.cu:
// 1176-1379).  The forward is in raster.cu.
//
// One 128-thread block per 16x16 tile; each of the 4 warps owns an 8x8 block
// and each lane two pixels of one column, four rows apart, so the
// per-Gaussian loop control and the warp reduction of the gradient terms are
// shared by 64 pixels (few tiles: 8 warps, one pixel per lane, kOnePixelTiles).
// Batches are staged and culled as in the forward: each record's mask of the
// blocks its cut ellipse can reach is found once, by the thread that stages it.
// The warps walk their records from the last contributor to the front, two at a
// time: both records' opacity terms are evaluated before the two transmittance
// recoveries so that their exp() chains overlap, and the two records' gradient
// vectors are summed in one warp reduction.  What bounds it: instruction issue
// (87 % with weights only, 79 % in the full adjoint).  At 1M Gaussians, 1080p:
// 0.364 -> 0.329 ms with the masks at staging and the exact skip threshold, ->
// 0.315 ms with T recovered by one approximate reciprocal and the exact-width
// reduction; full adjoint (500k, K = 5): 0.609 -> 0.581 -> 0.455 ms, also with
// the scalar recursion and the moments (adjoint_pixel).
#include "gsb_geometry.cuh"
#include "gsb_internal.h"
#include "gsb_tiles.cuh"

namespace gsb {

constexpr int kBatch = 256;

// Pixels of a lane: NP of one column, four rows apart.  NP = 2: 4 warps per
// tile, 8x8 pixels each; NP = 1: 8 warps, 8x4 pixels each.
template <int NP>
struct AdjLayout {
  static constexpr int kThreads = kTilePixels / NP;
  static constexpr int kRows = 4 * NP;             // rows of a warp's block
  static constexpr int kBands = kTile / kRows;     // of two blocks of 8 columns each
};

template <int K>
__device__ __forceinline__ void load_feats(const float4* srec, int j, float v2w, float* f) {
  f[0] = v2w;  // channel 0 sits in v1.w
#pragma unroll
  for (int k = 1; k < K; ++k) {
    const float4 q = srec[(2 + (k - 1) / 4) * kBatch + j];
    f[k] = ((k - 1) & 3) == 0 ? q.x : ((k - 1) & 3) == 1 ? q.y : ((k - 1) & 3) == 2 ? q.z : q.w;
  }
}

// Sum of N per-lane values over groups of 2 * OFF lanes, spread over the
// group's lanes: each exchange step halves the values a lane carries (lanes
// with the step's bit set keep the upper half), so 11 values take 6 + 3 + 2 + 1
// shuffles instead of the 8 + 4 + 2 + 1 of 16 padded ones.  Returns this lane's
// total; *idx is the value it holds, *owner is set on one lane per value and
// group.
template <int N, int OFF>
__device__ __forceinline__ float warp_spread_sum(float* x, int lane, int* idx, bool* owner) {
  constexpr int kHalf = (N + 1) / 2;
  const bool hi = (lane & OFF) != 0;
  if constexpr (N > 1) {
#pragma unroll
    for (int i = 0; i < kHalf; ++i) {
      const float other = kHalf + i < N ? x[kHalf + i < N ? kHalf + i : 0] : 0.f;
      x[i] = (hi ? other : x[i]) + __shfl_xor_sync(0xffffffffu, hi ? x[i] : other, OFF);
    }
    int at = 0;
    bool own = true;
    float v = x[0];
    if constexpr (OFF > 1)
      v = warp_spread_sum<kHalf, OFF / 2>(x, lane, &at, &own);
    else
      static_assert(N <= 2, "more values than lanes");
    *idx = at + (hi ? kHalf : 0);
    *owner = own && at < (hi ? N - kHalf : kHalf);
    return v;
  } else {
    float v = x[0];
#pragma unroll
    for (int o = OFF; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    *idx = 0;
    *owner = (lane & (2 * OFF - 1)) == 0;
    return v;
  }
}

// Per-pixel back-to-front state of the adjoint.
template <int K>
struct BwdPixel {
  float dl[K];
  float T, R;  // R: dl . (what is blended behind), the full adjoint's
  int cont;
};

// One contributor of one pixel in the adjoint: recovers T, accumulates the
// pixel's gradient terms into x: x[0..K) features, then (GEOM) alpha and the
// moments h d, h d d^T of h = dL/dalpha' alpha' (finish_geom).  With s = dl . f,
// dL/dalpha' = T (s - R), where R is the blended s of everything behind the
// record: one scalar recursion instead of one per channel (0.565 -> 0.481 ms
// at 500k Gaussians, 1080p, K = 5, with the moments).
template <int K, bool GEOM>
__device__ __forceinline__ bool adjoint_pixel(BwdPixel<K>& p, int idx, float m, float4 v1,
                                              float dx, float dy, const float* f, float* x) {
  if (!(idx < p.cont) || !(m >= v1.y)) return false;
  const float g = expf(m);
  const float ap = fminf(kAlphaMax, v1.z * g);
  p.T *= rcp_approx(1.f - ap);
  const float wgt = ap * p.T;
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] += p.dl[k] * wgt;
  if constexpr (GEOM) {
    float s = p.dl[0] * f[0];
#pragma unroll
    for (int k = 1; k < K; ++k) s += p.dl[k] * f[k];
    const float t = s - p.R;
    const float dap = p.T * t;
    p.R = fmaf(ap, t, p.R);
    const float h = dap * ap, tx = h * dx, ty = h * dy;
    x[K] += dap * g;
    x[K + 1] += tx;
    x[K + 2] += ty;
    x[K + 3] += tx * dx;
    x[K + 4] += tx * dy;
    x[K + 5] += ty * dy;
  }
  return true;
}

// The lane's moments to its centre (K + 1, K + 2) and conic gradients.
template <int K>
__device__ __forceinline__ void finish_geom(float4 v0, float4 v1, float* x) {
  const float Sx = x[K + 1], Sy = x[K + 2];
  x[K + 1] = 2.f * v0.z * Sx + v0.w * Sy;
  x[K + 2] = v0.w * Sx + 2.f * v1.x * Sy;
  x[K + 3] *= -0.5f;
  x[K + 4] = -x[K + 4];
  x[K + 5] *= -0.5f;
}

// Weights-only adjoint of two contributors at once: slot ja lies behind slot
// jb in list order, so it is undone first.  Both records' opacity terms are
// evaluated for both pixels before either transmittance update, so the four
// exp() chains overlap; the skip tests and the T recovery are exactly those
// of adjoint_pixel.  The two gradient vectors are summed together: one
// exchange at offset 16 leaves ja's partial sums on lanes 0-15 and jb's on
// lanes 16-31, then each half-warp spreads its K values (5 + 7 shuffles for
// K = 5).  When at most kDirectLanes lanes hit each record, those lanes add
// their own sums
// directly (at most 2 x kDirectLanes x K atomics instead of about 60
// reduction instructions; 47 % of the records a warp visits have so few hits
// at 1M Gaussians, 1080p).  Measured, near / far view: 4 lanes 0.367 / 0.282
// ms, 8 lanes 0.362 / 0.278, 12 lanes 0.360 / 0.275, 16 lanes 0.361 / 0.278.
constexpr int kDirectLanes = 12;
template <int K, int NP>
__device__ __forceinline__ void adjoint_weights_pair(BwdPixel<K> (&p)[NP], int base, int ja,
                                                     int jb, const float4* srec,
                                                     const int32_t* sgid, float fx,
                                                     const float (&fy)[NP], int lane,
                                                     float* __restrict__ dfeat) {
  const float4 a0 = srec[ja], a1 = srec[kBatch + ja];
  const float4 b0 = srec[jb], b1 = srec[kBatch + jb];
  float apa[NP], apb[NP];
  bool ua[NP], ub[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
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
  for (int q = 0; q < NP; ++q) {
    if (ua[q]) {
      p[q].T *= rcp_approx(1.f - apa[q]);
      const float wgt = apa[q] * p[q].T;
#pragma unroll
      for (int k = 0; k < K; ++k) xa[k] += p[q].dl[k] * wgt;
    }
  }
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    if (ub[q]) {
      p[q].T *= rcp_approx(1.f - apb[q]);
      const float wgt = apb[q] * p[q].T;
#pragma unroll
      for (int k = 0; k < K; ++k) xb[k] += p[q].dl[k] * wgt;
    }
  }
  const bool ha = ua[0] || ua[NP - 1], hb = ub[0] || ub[NP - 1];
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
  const bool hi = (lane & 16) != 0;
  float y[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float send = hi ? xa[k] : xb[k];
    const float keep = hi ? xb[k] : xa[k];
    y[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  int vidx;
  bool owner;
  const float tot = warp_spread_sum<K, 8>(y, lane, &vidx, &owner);
  if (owner && (hi ? cb : ca) != 0u) {
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
// 0-15 and jb's on lanes 16-31, then each half-warp spreads its values (11 + 12
// shuffles for K = 5).  When
// at most kDirectLanesGeom lanes hit each record, those lanes add their own
// K + 6 sums directly: at 1M / 1080p 0.776 -> 0.755 ms near, 0.462 -> 0.439
// ms far, against direct atomics for single hits only.
constexpr int kDirectLanesGeom = 8;
template <int K, int NP>
__device__ __forceinline__ void adjoint_geom_pair(BwdPixel<K> (&p)[NP], int base, int ja, int jb,
                                                  const float4* srec, const int32_t* sgid,
                                                  float fx, const float (&fy)[NP], int lane,
                                                  float* __restrict__ dfeat,
                                                  float* __restrict__ dalpha,
                                                  float* __restrict__ du,
                                                  float* __restrict__ dconic) {
  constexpr int NREAL = K + 6;
  const float4 a0 = srec[ja], a1 = srec[kBatch + ja];
  const float4 b0 = srec[jb], b1 = srec[kBatch + jb];
  float xa[NREAL], xb[NREAL];
#pragma unroll
  for (int v = 0; v < NREAL; ++v) xa[v] = xb[v] = 0.f;
  const float dxa = a0.x - fx, dxb = b0.x - fx;
  float dya[NP], dyb[NP], ma[NP], mb[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    dya[q] = a0.y - fy[q];
    dyb[q] = b0.y - fy[q];
    ma[q] = fminf(0.f, half_form(a0.z, a0.w, a1.x, dxa, dya[q]));
    mb[q] = fminf(0.f, half_form(b0.z, b0.w, b1.x, dxb, dyb[q]));
  }
  float fa[K], fb[K];
  load_feats<K>(srec, ja, a1.w, fa);
  load_feats<K>(srec, jb, b1.w, fb);
  bool ha = false, hb = false;
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    ha |= adjoint_pixel<K, true>(p[q], base + ja, ma[q], a1, dxa, dya[q], fa, xa);
    hb |= adjoint_pixel<K, true>(p[q], base + jb, mb[q], b1, dxb, dyb[q], fb, xb);
  }
  finish_geom<K>(a0, a1, xa);
  finish_geom<K>(b0, b1, xb);
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
  float y[NREAL];
#pragma unroll
  for (int v = 0; v < NREAL; ++v) {
    const float send = hi ? xa[v] : xb[v];
    const float keep = hi ? xb[v] : xa[v];
    y[v] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  int vidx;
  bool owner;
  const float tot = warp_spread_sum<NREAL, 8>(y, lane, &vidx, &owner);
  if (owner && (hi ? cb : ca) != 0u) {
    const int64_t g = sgid[hi ? jb : ja];
    atomicAdd(grad_slot<K>(vidx, g, dfeat, dalpha, du, dconic), tot);
  }
}

// Stages the records [base, base + cnt) of a tile's list, with their block masks.
template <int K, bool GEOM, int NP>
__device__ __forceinline__ void stage_batch(const int32_t* __restrict__ gsid,
                                            const float4* __restrict__ records, int first, int cnt,
                                            int X0, int Y0, float4* srec, int32_t* sgid,
                                            uint8_t* smask) {
  using L = AdjLayout<NP>;
  constexpr int V = RecordLayout<K>::kVec4;
  for (int t = threadIdx.x; t < cnt; t += L::kThreads) {
    const int g = gsid[first + t];
    const float4* src = records + (int64_t)g * V;
    const float4 v0 = __ldg(src), v1 = __ldg(src + 1), v2 = __ldg(src + 2);
    srec[t] = v0;
    srec[kBatch + t] = v1;
#pragma unroll
    for (int v = 3; v < V; ++v)
      if (GEOM) srec[(v - 1) * kBatch + t] = __ldg(src + v);
    sgid[t] = g;
    smask[t] = (uint8_t)region_mask<2, L::kBands, 8, L::kRows>(v0, v1, v2, X0, Y0);
  }
}

// Incoming gradients above this (infinite ones and NaN among them) leave the scalar
// recursion: dl . f would overflow, and inf - inf is NaN where the blended features
// of each channel stay finite and give signed infinities.  (A feature that is itself
// infinite gives its pixels' contributors infinite or NaN gradients either way.)
constexpr float kTame = 1e30f;
constexpr int kWild = 0x7fffffff;  // as a tile's largest contributor index

// Walks each pixel's contributors back to front from its `contrib` index,
// recovering T by division by (1 - alpha') from the saved final T.  The
// per-pixel skip decisions use the forward's exact expressions, so the walk
// visits exactly the Gaussians the forward blended; T itself is recovered
// with a fast reciprocal division (relative error ~1e-7 per step).  Per
// Gaussian each lane first adds its two pixels' terms, then the warp's 64
// pixels are summed with one transposed reduction and added with one atomic
// per value.  GEOM adds the opacity / centre / conic adjoint (draw_color_B's
// terms, for any channel count); dL/dT_final (vanilla_3dgs/gsplatcu/kernel.cu:
// 912-919) enters as the value of R behind the last contributor, since
// d T_final / d alpha' = -T_final / (1 - alpha').  As in the reference, the 0.99
// clamp and max(0, .) are not differentiated.  Weights-only at least 8 blocks of 128
// threads per SM (61 registers above 5 channels; 56 up to 5, where 9 fit); full
// adjoint 7 for K = 4 and 5 (500k: K = 4 0.513 against 0.519 ms at 6, K = 5 0.462
// against 0.476), 6 otherwise (K = 3: 0.364 against 0.371 ms at 7; above 5 channels 7
// would spill 90 bytes).
template <int K, bool GEOM, int NP>
__global__ void __launch_bounds__(AdjLayout<NP>::kThreads,
                                  (GEOM ? (K == 4 || K == 5 ? 7 : 6) : 8) * NP / 2)
    k_draw_backward(int H, int W, int gx, const int2* __restrict__ ranges,
                    const int32_t* __restrict__ gsid, const float4* __restrict__ records,
                    int32_t* __restrict__ order,
                    const int32_t* __restrict__ contrib, const float* __restrict__ final_tau,
                    const float* __restrict__ dout, const float* __restrict__ dtau,
                    float* __restrict__ dfeat, float* __restrict__ dalpha,
                    float* __restrict__ du, float* __restrict__ dconic) {
  pdl_wait();
  using L = AdjLayout<NP>;
  constexpr int V = RecordLayout<K>::kVec4;
  constexpr int NREAL = GEOM ? K + 6 : K;
  constexpr int kKeep = GEOM ? V - 1 : 2;  // float4s kept (v0, v1 and, with GEOM, the further channels)
  __shared__ float4 srec[kKeep * kBatch];
  __shared__ int32_t sgid[kBatch];
  __shared__ uint8_t smask[kBatch];
  __shared__ unsigned s_maxc;
  const int tile = order[blockIdx.x];
  if (tile < 0) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int X0 = (tile % gx) * kTile, Y0 = (tile / gx) * kTile;
  const int px = X0 + (w & 1) * 8 + (lane & 7);
  const int py = Y0 + (w >> 1) * L::kRows + (lane >> 3);
  const int2 rg = ranges[tile];
  if (rg.y - rg.x == 0) return;  // uniform per block
  const int64_t hw = (int64_t)H * W;
  BwdPixel<K> p[NP];
  float fy[NP];
  int wmax = 0;
  bool tame = true;
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const bool in = px < W && py + 4 * q < H;
    const int64_t pix = (int64_t)(py + 4 * q) * W + px;
    fy[q] = (float)(py + 4 * q);
#pragma unroll
    for (int k = 0; k < K; ++k) p[q].dl[k] = in ? dout[k * hw + pix] : 0.f;
    p[q].T = in ? final_tau[pix] : 0.f;
    p[q].R = (GEOM && dtau && in) ? dtau[pix] : 0.f;
    p[q].cont = in ? contrib[pix] : 0;
    wmax = max(wmax, p[q].cont);
    if constexpr (GEOM) {
#pragma unroll
      for (int k = 0; k < K; ++k) tame &= fabsf(p[q].dl[k]) <= kTame;
      tame &= fabsf(p[q].R) <= kTame;
    }
  }
  if (GEOM && !tame) wmax = kWild;
  wmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)wmax);
  if (threadIdx.x == 0) s_maxc = 0u;
  __syncthreads();
  if (lane == 0) atomicMax(&s_maxc, (unsigned)wmax);
  __syncthreads();
  if (GEOM && (int)s_maxc == kWild) {  // k_draw_backward_wild's
    if (threadIdx.x == 0) order[blockIdx.x] = ~tile;
    return;
  }
  // contributor indices never exceed the tile's list (clamped for safety
  // against mismatched inputs)
  const int maxc = min((int)s_maxc, rg.y - rg.x);
  const float fx = (float)px;
  for (int top = maxc; top > 0; top -= kBatch) {
    const int base = max(0, top - kBatch);
    const int cnt = top - base;
    __syncthreads();
    stage_batch<K, GEOM, NP>(gsid, records, rg.x + base, cnt, X0, Y0, srec, sgid, smask);
    __syncthreads();
    const int hi = min(cnt, wmax - base);
    for (int s_hi = hi; s_hi > 0; s_hi -= 32) {
      const int s_lo = max(0, s_hi - 32);
      const int j = s_lo + lane;
      unsigned mask = __ballot_sync(0xffffffffu, j < s_hi && ((smask[j] >> w) & 1));
      while (mask) {
        const int msb = 31 - __clz(mask);
        mask &= ~(1u << msb);
        if (mask) {
          const int msb2 = 31 - __clz(mask);
          mask &= ~(1u << msb2);
          if constexpr (GEOM)
            adjoint_geom_pair<K, NP>(p, base, s_lo + msb, s_lo + msb2, srec, sgid, fx, fy, lane,
                                       dfeat, dalpha, du, dconic);
          else
            adjoint_weights_pair<K, NP>(p, base, s_lo + msb, s_lo + msb2, srec, sgid, fx, fy, lane,
                                        dfeat);
          continue;
        }
        const int jj = s_lo + msb;
        const int idx = base + jj;
        float x[NREAL];
#pragma unroll
        for (int v = 0; v < NREAL; ++v) x[v] = 0.f;
        const float4 v0 = srec[jj];
        const float4 v1 = srec[kBatch + jj];
        const float dx = v0.x - fx;
        float f[K];
        if (GEOM) load_feats<K>(srec, jj, v1.w, f);
        bool hit = false;
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const float dy = v0.y - fy[q];
          const float m = fminf(0.f, half_form(v0.z, v0.w, v1.x, dx, dy));
          hit |= adjoint_pixel<K, GEOM>(p[q], idx, m, v1, dx, dy, f, x);
        }
        if constexpr (GEOM) finish_geom<K>(v0, v1, x);
        const unsigned cm = __ballot_sync(0xffffffffu, hit);
        if (!cm) continue;
        const int64_t g = sgid[jj];
        if (__popc(cm) == 1) {
          if (hit) {
#pragma unroll
            for (int v = 0; v < NREAL; ++v)
              atomicAdd(grad_slot<K>(v, g, dfeat, dalpha, du, dconic), x[v]);
          }
          continue;
        }
        int vidx;
        bool owner;
        const float tot = warp_spread_sum<NREAL, 16>(x, lane, &vidx, &owner);
        if (owner)
          atomicAdd(grad_slot<K>(vidx, g, dfeat, dalpha, du, dconic), tot);
      }
    }
  }
}

// Full adjoint of the tiles that k_draw_backward left out (kTame; it marks them in
// the launch order), with the features blended behind each record kept per channel:
// the terms as the reference forms them.  One pixel per thread.  A launch of its own,
// of kWildTiles tiles per block: as a call inside k_draw_backward it cost that kernel
// registers and 2 to 4 % (500k, 1080p, K = 5: 526 -> 537 us; K = 3: 424 -> 443).
constexpr int kWildTiles = 8;
template <int K>
__global__ void __launch_bounds__(kTilePixels)
    k_draw_backward_wild(int tiles, int H, int W, int gx, const int2* __restrict__ ranges,
                         const int32_t* __restrict__ gsid, const float4* __restrict__ records,
                         const int32_t* __restrict__ order, const int32_t* __restrict__ contrib,
                         const float* __restrict__ final_tau, const float* __restrict__ dout,
                         const float* __restrict__ dtau, float* __restrict__ dfeat,
                         float* __restrict__ dalpha, float* __restrict__ du,
                         float* __restrict__ dconic) {
  pdl_wait();
  using L = AdjLayout<1>;
  constexpr int NREAL = K + 6;
  __shared__ float4 srec[(RecordLayout<K>::kVec4 - 1) * kBatch];
  __shared__ int32_t sgid[kBatch];
  __shared__ uint8_t smask[kBatch];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t hw = (int64_t)H * W;
  for (int e = 0; e < kWildTiles; ++e) {  // (uniform per block)
    const int at = blockIdx.x * kWildTiles + e;
    if (at >= tiles || order[at] >= 0) continue;
    const int tile = ~order[at];
    const int X0 = (tile % gx) * kTile, Y0 = (tile / gx) * kTile;
    const int px = X0 + (w & 1) * 8 + (lane & 7), py = Y0 + (w >> 1) * L::kRows + (lane >> 3);
    const bool in = px < W && py < H;
    const int64_t pix = (int64_t)py * W + px;
    const int2 rg = ranges[tile];
    const int n = rg.y - rg.x;
    float dl[K], G[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      dl[k] = in ? dout[k * hw + pix] : 0.f;
      G[k] = 0.f;
    }
    const float Tf = in ? final_tau[pix] : 0.f, dTf = (dtau && in) ? dtau[pix] : 0.f;
    const int cont = in ? contrib[pix] : 0;
    float T = Tf;
    for (int base = (n - 1) / kBatch * kBatch; base >= 0; base -= kBatch) {
      const int cnt = min(kBatch, n - base);
      __syncthreads();
      stage_batch<K, true, 1>(gsid, records, rg.x + base, cnt, X0, Y0, srec, sgid, smask);
      __syncthreads();
      for (int j = cnt - 1; j >= 0; --j) {
        if (!((smask[j] >> w) & 1)) continue;  // (uniform per warp)
        const float4 v0 = srec[j], v1 = srec[kBatch + j];
        const float dx = v0.x - (float)px, dy = v0.y - (float)py;
        const float m = fminf(0.f, half_form(v0.z, v0.w, v1.x, dx, dy));
        const bool hit = base + j < cont && m >= v1.y;
        if (!__any_sync(0xffffffffu, hit)) continue;
        float f[K], x[NREAL];
        load_feats<K>(srec, j, v1.w, f);
#pragma unroll
        for (int v = 0; v < NREAL; ++v) x[v] = 0.f;
        if (hit) {
          const float g = expf(m), ap = fminf(kAlphaMax, v1.z * g);
          const float one_m = 1.f - ap, inv = rcp_approx(one_m);
          T *= inv;
          float dap = 0.f;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            x[k] = dl[k] * (ap * T);
            dap += dl[k] * (T * (f[k] - G[k]));
            G[k] = ap * f[k] + one_m * G[k];
          }
          if (dtau) dap += dTf * (-Tf * inv);
          x[K] = dap * g;
          x[K + 1] = dap * ((2.f * v0.z * dx + v0.w * dy) * ap);
          x[K + 2] = dap * ((v0.w * dx + 2.f * v1.x * dy) * ap);
          x[K + 3] = dap * (-0.5f * ap * (dx * dx));
          x[K + 4] = dap * (-1.0f * ap * (dx * dy));
          x[K + 5] = dap * (-0.5f * ap * (dy * dy));
        }
        int vidx;
        bool owner;
        const float tot = warp_spread_sum<NREAL, 16>(x, lane, &vidx, &owner);
        if (owner) atomicAdd(grad_slot<K>(vidx, sgid[j], dfeat, dalpha, du, dconic), tot);
      }
    }
  }
}

// Up to this many tiles (4 blocks for each of 148 SMs) a warp is alone on its
// scheduler or nearly so, and the time is the longest tile's chain of records: with
// one pixel per lane it is shorter.  Two pixels / one, K = 5: 256 tiles, 20k Gaussians
// 102 / 66 us (weights only 66 / 47), 80k 336 / 209; 432 tiles, 40k 168 / 109; 600
// tiles, 60k 221 / 141, 240k 397 / 265.  On larger images the instructions count, 1.35x
// as many, and the outcome depends on how long the longest list is: 1200 tiles, 600k
// 385 / 308; 1900, 600k 367 / 371; 3600, 250k 285 / 261, 1M 455 / 531; 4346, 300k
// 290 / 360; 8160, 1M weights only 315 / 429.  The line lies where one pixel always won.
constexpr int kOnePixelTiles = 592;

template <int K>
static void draw_bwd_k(int tiles, int H, int W, int gx, const int2* rg, const int32_t* gsid,
                       const float4* rec, int32_t* order, const int32_t* contrib,
                       const float* ft, const float* dout, const float* dtau, float* dfeat,
                       float* dalpha, float* du, float* dq, cudaStream_t st) {
  const bool one = tiles <= kOnePixelTiles;
  auto kern = one ? (dalpha ? k_draw_backward<K, true, 1> : k_draw_backward<K, false, 1>)
                  : (dalpha ? k_draw_backward<K, true, 2> : k_draw_backward<K, false, 2>);
  launch_pdl(kern, dim3(tiles), dim3(kTilePixels / (one ? 1 : 2)), 0, st, H, W, gx, rg, gsid, rec,
             order, contrib, ft, dout, dtau, dfeat, dalpha, du, dq);
  if (dalpha)
    launch_pdl(k_draw_backward_wild<K>, dim3(div_up(tiles, kWildTiles)), dim3(kTilePixels), 0, st,
               tiles, H, W, gx, rg, gsid, rec, (const int32_t*)order, contrib, ft, dout, dtau, dfeat,
               dalpha, du, dq);
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
  return check_launch("splat_backward", dalpha ? 2 : 1);
}

}  // namespace gsb
