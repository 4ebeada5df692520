// The differentiation workload's loss in one kernel: the palette colour image
// img_c = sum_k palette[k][c] layer_k, the L1 + SSIM loss of gau_loss
// (vanilla_3dgs/gsplat/pytorch_ssim.py:26-67) against a target, the
// negative-weight penalty of finetune.py:375,381, and the gradient of all of
// it w.r.t. the layer stack and the palette.
//
// SSIM's gradient at a pixel q needs the SSIM partials at every pixel within
// the window radius R = 5 of q, and each partial needs the window statistics
// (means, second moments) of the pixels within R of it.  The 11x11 Gaussian
// window is applied as two 11-tap passes (it is the outer product of the 1-D
// Gaussian).  A block walks down a strip of 32 output columns and all three
// channels, eleven rows a step:
//   H1  the rows' horizontal statistics, 42 columns, six outputs per thread;
//   V1  one thread per column and channel keeps the eleven window sums that are
//       open at a time in registers; each row closes one, which gives the SSIM
//       map and its partials five rows further up;
//   H2  the partials' horizontal pass, 32 columns, four outputs per thread;
//   V2  as V1, giving d loss / d image another five rows up; then the layer and
//       palette gradients, a pixel per thread.
// H1 and H2 are shared by all threads; V1 is half the block's work while the
// other half does V2 of the step before and the gradients.  A row's horizontal
// passes are computed once per strip and its vertical sums read each value once;
// only the columns' halo and the 20 rows around a strip's segment are computed
// twice.  The loss and its full gradient come out of one launch (the gradient of
// a mean does not depend on the loss value).
//
// The statistics are (mean x, mean y) and (mean x^2 + y^2, mean xy): SSIM needs
// the two variances only as a sum.  Each pair is one packed FMA per tap.
//
// What bounds it: issue (half of the slots; the rest is the barriers between the
// passes, with three blocks per SM to fill them).  32x32 tiles that recomputed
// their halo on every side and passed every sum through shared memory took
// 0.220 ms at 1080p, K = 5, 0.113 at 720p and 0.024 at 256^2; this takes 0.134,
// 0.069 and 0.017 (the form for a block alone).  Two blocks per SM without spills 0.164; staging and gradients
// on a third group of threads 0.176; a rolled row loop 0.16.
#include <algorithm>
#include <cmath>

#include "gsb_common.cuh"
#include "gsb_internal.h"

namespace gsb {

constexpr int kSsimR = 5;                        // window radius
constexpr int kSsimTaps = 2 * kSsimR + 1;
constexpr int kSsimW = 32;                       // output columns of a strip
constexpr int kSsimMW = kSsimW + 2 * kSsimR;     // 42: columns with statistics
constexpr int kSsimXW = kSsimW + 4 * kSsimR;     // 52: columns staged
constexpr int kSsimStep = 11;                    // rows of a step
constexpr int kSsimRows = 3 * kSsimStep;         // rows of a step, all channels
constexpr int kSsimRole = 128, kSsimThreads = 2 * kSsimRole;
constexpr int kSsimBlocks = 3;                   // resident blocks per SM (66 KB, 80 registers)
constexpr int kRunH1 = 6, kRunH2 = 4;            // outputs per thread, horizontal passes
constexpr int kItemsH1 = kSsimRows * (kSsimMW / kRunH1);  // 231
constexpr int kItemsH2 = kSsimRows * (kSsimW / kRunH2);   // 264
static_assert(kSsimMW % kRunH1 == 0 && kSsimW % kRunH2 == 0, "runs");
static_assert(3 * kSsimMW <= kSsimRole && 3 * kSsimW <= kSsimRole, "one thread per column");
// Row pitches in 16-byte units: odd, so that eight threads on eight rows read
// and write eight different groups of banks.
constexpr int kPitchXY = 27, kPitchH = 43, kPitchMa = 21, kPitchMb = 11, kPitchGa = 17,
              kPitchGb = 9;
constexpr size_t kSsimSmemBytes =
    (size_t)kSsimRows * (kPitchXY + kPitchH + kPitchMa + kPitchMb + kPitchGa + kPitchGb) * 16;

// Two FP32 values in one 64-bit register; each half rounds as the scalar operation.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct SsimWindow {
  float g[kSsimTaps];  // symmetric
};

struct SsimScales {
  float c1, c2;    // (0.01 range)^2, (0.03 range)^2
  float inv_n;     // 1 / (3 H W)
  float w_l1;      // (1 - lambda_ssim) / (3 H W)
  float w_ssim;    // lambda_ssim / (3 H W)
  float w_pos;     // lambda_pos / (K H W)
  float lambda_ssim;
};

__global__ void k_l1_ssim_init(float* __restrict__ loss, float* __restrict__ dpal, int n_pal) {
  pdl_wait();
  if (threadIdx.x < 4) loss[threadIdx.x] = 0.f;
  if (dpal && threadIdx.x < n_pal) dpal[threadIdx.x] = 0.f;
}

// H1 of one item: six columns of one row and channel.
__device__ __forceinline__ void ssim_h1(const ulonglong2* sXY, ulonglong2* sH, const f32x2* g,
                                        int e) {
  const int run = e / kSsimRows, rr = e - run * kSsimRows;
  const ulonglong2* in = sXY + rr * kPitchXY + run * (kRunH1 / 2);
  f32x2 m[kRunH1], q[kRunH1];
#pragma unroll
  for (int o = 0; o < kRunH1; ++o) m[o] = q[o] = 0;
#pragma unroll
  for (int k = 0; k < (kRunH1 + 2 * kSsimR) / 2; ++k) {
    const ulonglong2 two = in[k];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const f32x2 v = h ? two.y : two.x;
      const float2 xy = unpack2(v);
      const f32x2 p = pack2(fmaf(xy.x, xy.x, xy.y * xy.y), xy.x * xy.y);
#pragma unroll
      for (int o = 0; o < kRunH1; ++o) {
        const int i = 2 * k + h - o;
        if (i >= 0 && i < kSsimTaps) {
          const int w = i <= kSsimR ? i : 2 * kSsimR - i;
          m[o] = fma2(g[w], v, m[o]);
          q[o] = fma2(g[w], p, q[o]);
        }
      }
    }
  }
  ulonglong2* out = sH + rr * kPitchH + run * kRunH1;
#pragma unroll
  for (int o = 0; o < kRunH1; ++o) out[o] = make_ulonglong2(m[o], q[o]);
}

// H2 of one item: four columns of one row and channel.
__device__ __forceinline__ void ssim_h2(const ulonglong2* sMa, const float4* sMb, ulonglong2* sGa,
                                        float4* sGb, const f32x2* g, int e) {
  const int run = e / kSsimRows, rr = e - run * kSsimRows;
  const ulonglong2* ia = sMa + rr * kPitchMa + run * (kRunH2 / 2);
  const float4* ib = sMb + rr * kPitchMb + run * (kRunH2 / 4);
  constexpr int kIn = kRunH2 + 2 * kSsimR;  // 14
  f32x2 a[kRunH2];
  float b[kRunH2], vb[kIn];
#pragma unroll
  for (int o = 0; o < kRunH2; ++o) a[o] = 0, b[o] = 0.f;
#pragma unroll
  for (int k = 0; k < kIn / 4; ++k) {
    const float4 v = ib[k];
    vb[4 * k] = v.x, vb[4 * k + 1] = v.y, vb[4 * k + 2] = v.z, vb[4 * k + 3] = v.w;
  }
  {
    const float2 v = *reinterpret_cast<const float2*>(ib + kIn / 4);
    vb[kIn - 2] = v.x, vb[kIn - 1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < kIn / 2; ++k) {
    const ulonglong2 two = ia[k];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const f32x2 v = h ? two.y : two.x;
#pragma unroll
      for (int o = 0; o < kRunH2; ++o) {
        const int i = 2 * k + h - o;
        if (i >= 0 && i < kSsimTaps) {
          const int w = i <= kSsimR ? i : 2 * kSsimR - i;
          a[o] = fma2(g[w], v, a[o]);
          b[o] = fmaf(unpack2(g[w]).x, vb[2 * k + h], b[o]);
        }
      }
    }
  }
  ulonglong2* oa = sGa + rr * kPitchGa + run * (kRunH2 / 2);
  oa[0] = make_ulonglong2(a[0], a[1]);
  oa[1] = make_ulonglong2(a[2], a[3]);
  sGb[rr * kPitchGb + run] = make_float4(b[0], b[1], b[2], b[3]);
}

// Stages a step: the image (from one read of the layer stack) and the target,
// as (x, y) pairs, zero outside the image.  First image row `top`, column `left`.
template <int K, bool ALONE>
__device__ __forceinline__ void ssim_stage(float2* sXY, const float* __restrict__ layer,
                                           const float* __restrict__ target, const float* sP,
                                           int H, int W, int64_t hw, int top, int left, int t) {
#pragma unroll (ALONE ? 3 : 1)
  for (int u = 0; u < (kSsimStep * kSsimXW + kSsimThreads - 1) / kSsimThreads; ++u) {
    const int e = t + u * kSsimThreads;
    if (e >= kSsimStep * kSsimXW) break;
    const int r = e / kSsimXW, q = e - r * kSsimXW;
    const int iy = top + r, ix = left + q;
    const bool in = iy >= 0 && iy < H && ix >= 0 && ix < W;
    const int64_t p = in ? (int64_t)iy * W + ix : 0;
    float l[K], y[3];
#pragma unroll
    for (int k = 0; k < K; ++k) l[k] = in ? layer[k * hw + p] : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) y[c] = in ? target[c * hw + p] : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float x = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) x = fmaf(sP[3 * k + c], l[k], x);
      sXY[(c * kSsimStep + r) * (2 * kPitchXY) + q] = make_float2(x, y[c]);
    }
  }
}

// Barrier of `Threads` threads that come to it from either role's loop.
template <int Id, int Threads>
__device__ __forceinline__ void ssim_sync() {
  asm volatile("barrier.sync %0, %1;" ::"n"(Id), "n"(Threads) : "memory");
}

// Grid: strips x segments of `rows` output rows each.  ALONE: a grid of at most one
// block per SM, whose time is one block's chain of steps: it may use all registers and
// has the loads of a step's staging and gradients in flight together.
template <int K, bool PAL, bool ALONE>
__global__ void __launch_bounds__(kSsimThreads, ALONE ? 1 : kSsimBlocks)
    k_palette_l1_ssim(int H, int W, int rows, const float* __restrict__ layer,
                      const float* __restrict__ palette, const float* __restrict__ target,
                      SsimWindow win, SsimScales sc, float* __restrict__ image,
                      float* __restrict__ loss, float* __restrict__ dlayer,
                      float* __restrict__ dpal) {
  pdl_wait();
  extern __shared__ float4 smem[];
  float4* sp = smem;
  ulonglong2* sXY = reinterpret_cast<ulonglong2*>(sp);  // (x, y), 52 columns
  sp += kSsimRows * kPitchXY;
  ulonglong2* sH = reinterpret_cast<ulonglong2*>(sp);   // four statistics, 42 columns
  sp += kSsimRows * kPitchH;
  ulonglong2* sMa = reinterpret_cast<ulonglong2*>(sp);  // partials w.r.t. mu_x and s_xx
  sp += kSsimRows * kPitchMa;
  float4* sMb = sp;                                     // partial w.r.t. s_xy
  sp += kSsimRows * kPitchMb;
  ulonglong2* sGa = reinterpret_cast<ulonglong2*>(sp);  // the same, filtered
  sp += kSsimRows * kPitchGa;
  float4* sGb = sp;
  __shared__ float sP[3 * K];
  __shared__ float red[kSsimThreads / 32][3 + 3 * K];

  const int tid = threadIdx.x, role = tid / kSsimRole, t = tid % kSsimRole;
  const int x0 = blockIdx.x * kSsimW, y0 = blockIdx.y * rows;
  const int y1 = min(y0 + rows, H);
  const int64_t hw = (int64_t)H * W;
  const int steps = (y1 - y0 + 4 * kSsimR + kSsimStep - 1) / kSsimStep;
  f32x2 g[kSsimR + 1];
#pragma unroll
  for (int i = 0; i <= kSsimR; ++i) g[i] = pack2(win.g[i], win.g[i]);
  if (tid < 3 * K) sP[tid] = PAL ? palette[tid] : (tid / 3 == tid % 3 ? 1.f : 0.f);
  __syncthreads();

  // both roles' share of the horizontal passes: rows of step s and partials of
  // step s - 1
  auto horizontal = [&](int s) {
    if (s < steps)
#pragma unroll 1
      for (int e = tid; e < kItemsH1; e += kSsimThreads) ssim_h1(sXY, sH, g, e);
    if (s > 0)
#pragma unroll 1
      for (int e = tid; e < kItemsH2; e += kSsimThreads) ssim_h2(sMa, sMb, sGa, sGb, g, e);
  };
  ssim_stage<K, ALONE>(reinterpret_cast<float2*>(sXY), layer, target, sP, H, W, hw, y0 - 2 * kSsimR,
                x0 - 2 * kSsimR, tid);
  auto sync = [] { ssim_sync<0, kSsimThreads>(); };
  const int lane = tid & 31, w = tid >> 5;

  if (role == 0) {
    // V1: thread (c, j); the window sum that closes at row r of a step is slot r
    const bool on = t < 3 * kSsimMW;
    const int c = on ? t / kSsimMW : 0, j = on ? t - c * kSsimMW : 0;
    const int ix = x0 - kSsimR + j;
    const bool col_in = ix >= 0 && ix < W;
    const bool col_out = j >= kSsimR && j < kSsimR + kSsimW;
    f32x2 m[kSsimTaps], q[kSsimTaps];
#pragma unroll
    for (int k = 0; k < kSsimTaps; ++k) m[k] = q[k] = 0;
    float ssum = 0.f;
    sync();
    for (int s = 0; s <= steps; ++s) {
      horizontal(s);
      sync();
      if (s < steps && on) {
        const ulonglong2* in = sH + c * kSsimStep * kPitchH + j;
        float2* oa = reinterpret_cast<float2*>(sMa + c * kSsimStep * kPitchMa) + j;
        float* ob = reinterpret_cast<float*>(sMb + c * kSsimStep * kPitchMb) + j;
        const int top = y0 - 3 * kSsimR + s * kSsimStep;  // image row of the sums closing at r = 0
#pragma unroll
        for (int r = 0; r < kSsimStep; ++r) {
          const ulonglong2 v = in[r * kPitchH];
#pragma unroll
          for (int i = 0; i < kSsimTaps; ++i) {  // sum i closes i rows below
            const int k = i <= kSsimR ? i : 2 * kSsimR - i;
            m[i] = fma2(g[k], v.x, i + 1 < kSsimTaps ? m[i + 1] : 0);
            q[i] = fma2(g[k], v.y, i + 1 < kSsimTaps ? q[i + 1] : 0);
          }
          const int iy = top + r;
          float dm = 0.f, dxx = 0.f, dxy = 0.f;
          if (col_in && iy >= 0 && iy < H) {
            const float2 mu = unpack2(m[0]), sq = unpack2(q[0]);
            const float mx = mu.x, my = mu.y;
            const float mxy = mx * my, mm = fmaf(mx, mx, my * my);
            const float A1 = 2.f * mxy + sc.c1;
            const float A2 = 2.f * (sq.y - mxy) + sc.c2;
            const float B1 = mm + sc.c1;
            const float B2 = (sq.x - mm) + sc.c2;
            // B1 >= C1 > 0 and B2 > 0 up to rounding: the fast reciprocal's
            // relative error (2 ulp) is far below the gradient tolerance
            const float rB1 = __fdividef(1.f, B1), rB2 = __fdividef(1.f, B2);
            const float inv = rB1 * rB2;
            const float S = A1 * A2 * inv;
            dm = 2.f * my * (A2 - A1) * inv - 2.f * mx * S * (rB1 - rB2);
            dxx = -S * rB2;
            dxy = 2.f * A1 * inv;
            if (col_out && iy >= y0 && iy < y1) ssum += S;
          }
          oa[r * (2 * kPitchMa)] = make_float2(dm, dxx);
          ob[r * (4 * kPitchMb)] = dxy;
        }
      }
      if (s + 1 < steps)
        ssim_stage<K, ALONE>(reinterpret_cast<float2*>(sXY), layer, target, sP, H, W, hw,
                      y0 - 2 * kSsimR + (s + 1) * kSsimStep, x0 - 2 * kSsimR, tid);
      sync();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, o);
    if (lane == 0) red[w][1] = ssum;
  } else {
    // V2: thread (c, tx), then one pixel per thread; stages the next step's rows
    const int c = t / kSsimW, tx = t % kSsimW, gx = x0 + tx;
    f32x2 a[kSsimTaps];
    float b[kSsimTaps];
#pragma unroll
    for (int k = 0; k < kSsimTaps; ++k) a[k] = 0, b[k] = 0.f;
    float l1 = 0.f, pen = 0.f, dp[K][3];
#pragma unroll
    for (int k = 0; k < K; ++k) dp[k][0] = dp[k][1] = dp[k][2] = 0.f;
    sync();
    for (int s = 0; s <= steps; ++s) {
      horizontal(s);
      sync();
      if (s > 0) {
        if (c < 3) {
          f32x2* ga = reinterpret_cast<f32x2*>(sGa + c * kSsimStep * kPitchGa) + tx;
          float* gb = reinterpret_cast<float*>(sGb + c * kSsimStep * kPitchGb) + tx;
#pragma unroll
          for (int r = 0; r < kSsimStep; ++r) {
            const f32x2 va = ga[r * (2 * kPitchGa)];
            const float vb = gb[r * (4 * kPitchGb)];
#pragma unroll
            for (int i = 0; i < kSsimTaps; ++i) {
              const int k = i <= kSsimR ? i : 2 * kSsimR - i;
              a[i] = fma2(g[k], va, i + 1 < kSsimTaps ? a[i + 1] : 0);
              b[i] = fmaf(unpack2(g[k]).x, vb, i + 1 < kSsimTaps ? b[i + 1] : 0.f);
            }
            ga[r * (2 * kPitchGa)] = a[0];  // over this thread's own inputs
            gb[r * (4 * kPitchGb)] = b[0];
          }
        }
        ssim_sync<1, kSsimRole>();
        const int top = y0 - 4 * kSsimR + (s - 1) * kSsimStep;  // output row of r = 0
#pragma unroll (ALONE ? 3 : 1)
        for (int u = 0; u < 3; ++u) {
          const int r = t / kSsimW + 4 * u, gy = top + r;
          if (r < kSsimStep && gx < W && gy >= y0 && gy < y1) {
            const int64_t p = (int64_t)gy * W + gx;
            float l[K], y[3], dx[3];
#pragma unroll
            for (int k = 0; k < K; ++k) l[k] = layer[k * hw + p];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) y[cc] = target[cc * hw + p];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
              const int rr = cc * kSsimStep + r;
              const float2 ga = reinterpret_cast<const float2*>(sGa + rr * kPitchGa)[tx];
              const float gb = reinterpret_cast<const float*>(sGb + rr * kPitchGb)[tx];
              float x = 0.f;
#pragma unroll
              for (int k = 0; k < K; ++k) x = fmaf(sP[3 * k + cc], l[k], x);
              const float dS = ga.x + 2.f * x * ga.y + y[cc] * gb;
              const float d = x - y[cc];
              l1 += fabsf(d);
              const float sg = d > 0.f ? 1.f : (d < 0.f ? -1.f : 0.f);
              dx[cc] = sc.w_l1 * sg - sc.w_ssim * dS;
              if (image) image[cc * hw + p] = x;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
              pen += fmaxf(-l[k], 0.f);
              float gl = l[k] < 0.f ? -sc.w_pos : 0.f;
#pragma unroll
              for (int cc = 0; cc < 3; ++cc) {
                gl = fmaf(sP[3 * k + cc], dx[cc], gl);
                dp[k][cc] = fmaf(l[k], dx[cc], dp[k][cc]);
              }
              if (dlayer) dlayer[k * hw + p] = gl;
            }
          }
        }
      }
      if (s + 1 < steps)
        ssim_stage<K, ALONE>(reinterpret_cast<float2*>(sXY), layer, target, sP, H, W, hw,
                      y0 - 2 * kSsimR + (s + 1) * kSsimStep, x0 - 2 * kSsimR, tid);
      sync();
    }
    float v[2 + 3 * K];
    v[0] = l1;
    v[1] = pen;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      v[2 + 3 * k] = dp[k][0];
      v[3 + 3 * k] = dp[k][1];
      v[4 + 3 * k] = dp[k][2];
    }
#pragma unroll
    for (int k = 0; k < 2 + 3 * K; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
      if (lane == 0) red[w][k ? k + 1 : 0] = v[k];
    }
  }
  __syncthreads();
  // sums over the block: the SSIM sum from the first role's warps, all else from
  // the second's
  if (tid < 3 + 3 * K) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kSsimRole / 32; ++k) v += red[(tid == 1 ? 0 : kSsimRole / 32) + k][tid];
    if (tid < 3)
      atomicAdd(loss + 1 + tid, v * (tid == 2 ? sc.w_pos : sc.inv_n));
    else if (dpal)
      atomicAdd(dpal + (tid - 3), v);
    __threadfence();
  }
  __syncthreads();
  // The block that finishes last forms the total from the three sums: a total
  // added up block by block would round three times as often, at a larger value.
  // Until then loss[0] counts the blocks.
  if (tid == 0 && atomicAdd(reinterpret_cast<unsigned*>(loss), 1u) ==
                      gridDim.x * gridDim.y - 1) {
    __threadfence();
    const volatile float* part = loss;
    loss[0] = (float)((double)sc.lambda_ssim * (1.0 - (double)part[2]) +
                      (1.0 - (double)sc.lambda_ssim) * (double)part[1] + (double)part[3]);
  }
}

template <int K, bool PAL, bool ALONE>
static int launch_l1_ssim_k(dim3 grid, int rows, const float* layer, const float* palette,
                            const float* target, int H, int W, const SsimWindow& win,
                            const SsimScales& sc, float* image, float* loss, float* dlayer,
                            float* dpal, cudaStream_t st) {
  // opt in to > 48 KB of dynamic shared memory, once per device
  static bool attr[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr[dev]) {
    if (cudaFuncSetAttribute(k_palette_l1_ssim<K, PAL, ALONE>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kSsimSmemBytes) != cudaSuccess)
      return check_launch("palette_l1_ssim (shared memory attribute)", 0);
    if (dev >= 0 && dev < 64) attr[dev] = true;
  }
  launch_pdl(k_palette_l1_ssim<K, PAL, ALONE>, grid, dim3(kSsimThreads), kSsimSmemBytes, st, H, W,
             rows, layer, palette, target, win, sc, image, loss, dlayer, dpal);
  return check_launch("palette_l1_ssim");
}

int launch_palette_l1_ssim(int K, int H, int W, const float* layer, const float* palette,
                           const float* target, float lambda_ssim, float lambda_pos,
                           float data_range, float* image, float* loss, float* dlayer,
                           float* dpal, cudaStream_t st) {
  // the reference's window: the 1-D Gaussian rounded to FP32, divided by its
  // FP32 sum (pytorch_ssim.py:12-14)
  SsimWindow win;
  double e[kSsimTaps], sum = 0.0;
  for (int i = 0; i < kSsimTaps; ++i) {
    const double x = i - kSsimR;
    e[i] = (double)(float)std::exp(-x * x / (2.0 * 1.5 * 1.5));
    sum += e[i];
  }
  const float fsum = (float)sum;
  for (int i = 0; i < kSsimTaps; ++i) win.g[i] = (float)e[i] / fsum;
  const int64_t hw = (int64_t)H * W;
  SsimScales sc;
  sc.c1 = (0.01f * data_range) * (0.01f * data_range);
  sc.c2 = (0.03f * data_range) * (0.03f * data_range);
  sc.inv_n = hw ? (float)(1.0 / (3.0 * (double)hw)) : 0.f;
  sc.w_l1 = (1.f - lambda_ssim) * sc.inv_n;
  sc.w_ssim = lambda_ssim * sc.inv_n;
  sc.lambda_ssim = lambda_ssim;
  sc.w_pos = hw ? (float)((double)lambda_pos / ((double)K * (double)hw)) : 0.f;
  // an empty image has no pixels to average: its loss and gradients are 0
  launch_pdl(k_l1_ssim_init, dim3(1), dim3(32), 0, st, loss, dpal, 3 * K);
  int rc = check_launch("palette_l1_ssim (init)");
  if (rc || hw == 0) return rc;
  // Segments of 11 s - 20 rows take s steps and one to finish; the blocks that
  // are resident at a time run in waves.  Take the s of the least waves x steps.
  // Images whose segments of at most kAloneSteps steps fit on one block per SM take
  // the fewest such steps instead, in the form for a block alone: three blocks that
  // share an SM lengthen each other's steps, and at 80 registers they spill.  Shared /
  // alone, K = 5 and 8: 100x100 15.2, 17.3 / 13.9, 14.0 us; 257x257 21.2, 24.8 / 17.2,
  // 18.5; 300x300 21.4, 25.0 / 18.2, 20.3; 400x400 26.9, 32.0 / 25.0, 28.0; 2000x33
  // 26.5, 30.4 / 21.2, 22.9 (32x32 tiles, one per SM here, took 21.3, 22.9).  With more
  // steps the shared form wins: 640x480 32.9 / 35.8, 800x600 44.1 / 52.0.
  constexpr int kAloneSteps = 6;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t strips = (W + kSsimW - 1) / kSsimW, slots = (int64_t)sms * kSsimBlocks;
  const auto segments = [H](int s) {
    const int r = kSsimStep * s - 4 * kSsimR;
    return ((int64_t)H + r - 1) / r;
  };
  constexpr int kLeast = 4 * kSsimR / kSsimStep + 1;
  int steps = kLeast;
  while (steps < kAloneSteps && strips * segments(steps) > sms) ++steps;
  const bool alone = strips * segments(steps) <= sms;
  if (!alone) {
    int64_t best = -1;
    for (int s = kLeast;; ++s) {
      const int64_t segs = segments(s), cost = (strips * segs + slots - 1) / slots * (2 * s + 3);
      if (segs <= 65535 && (best < 0 || cost < best)) best = cost, steps = s;
      if (segs == 1) break;
    }
  }
  const int rows = kSsimStep * steps - 4 * kSsimR;
  const dim3 grid((unsigned)strips, (unsigned)((H + rows - 1) / rows));
  if (!palette)
    return (alone ? launch_l1_ssim_k<3, false, true> : launch_l1_ssim_k<3, false, false>)(
        grid, rows, layer, nullptr, target, H, W, win, sc, image, loss, dlayer, nullptr, st);
  switch (K) {
#define GSB_K(KK)                                                                          \
  case KK:                                                                                 \
    return (alone ? launch_l1_ssim_k<KK, true, true> : launch_l1_ssim_k<KK, true, false>)(  \
        grid, rows, layer, palette, target, H, W, win, sc, image, loss, dlayer, dpal, st);
    GSB_K(1) GSB_K(2) GSB_K(3) GSB_K(4) GSB_K(5) GSB_K(6) GSB_K(7) GSB_K(8)
#undef GSB_K
    default: return GSB_ERR_INVALID_ARGUMENT;
  }
}

}  // namespace gsb
