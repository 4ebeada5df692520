// Tile compositing, forward (draw_weight / draw_color, gsplatcu/kernel.cu:
// 194-372).  The adjoint is in raster_backward.cu.
//
// One 256-thread block per 16x16 tile; each of the 8 warps owns an 8x4 block
// of pixels, one per lane.  The tile's Gaussian list is staged through shared
// memory in batches of 256 packed records, each thread loading a whole record
// and finding which warps' blocks its cut ellipse can reach (region_mask,
// gsb_tiles.cuh).  The warps walk the records whose mask has their bit, in
// list order, two at a time: both records' opacity terms are evaluated before
// the two blends so that their exp() chains overlap.  Per pixel, a record
// beyond its skip threshold is not blended -- exactly the records the
// reference skips (alpha' < 0.002, gsb_record.cuh) -- and every other record is
// evaluated with the reference's own FP32 expressions, so skip/stop decisions,
// contributor indices and blended values agree with it.  What bounds it: FP32
// and special-function issue.  At 1M Gaussians, 1080p: 0.284 -> 0.245 ms with
// the masks found at staging and the exact skip threshold in the record (one
// comparison instead of two, no scaling of the form); 3M, 4K: 0.99 -> 0.88 ms.
#include "gsb_geometry.cuh"
#include "gsb_internal.h"
#include "gsb_tiles.cuh"

namespace gsb {

constexpr int kBatch = 256;
constexpr int kDrawThreads = 256;  // one pixel per thread, 8x4 pixels per warp

// ------------------------------------------------------ tile launch order
// Blocks are launched in blockIdx order, a wave at a time.  Compositing a
// tile costs roughly its list length, which varies by orders of magnitude
// across an image, so launching tiles in raster order leaves the last waves
// waiting on a few long tiles.  The compositing kernels instead take their
// tile from a launch order, longest list first (a largest-first schedule):
// lengths binned at a quarter octave, descending; order within a bin is
// arbitrary.  Measured at 1M Gaussians, 1080p: forward 0.309 -> 0.280 ms,
// adjoint 0.436 -> 0.372 ms (0.220 -> 0.164 and 0.317 -> 0.273 ms for a
// distant view).  The results do not depend on the order.
constexpr int kOrderThreads = 1024, kOrderBins = 128;

__device__ __forceinline__ int order_bin(int2 rg) {
  const uint32_t x = (uint32_t)max(0, rg.y - rg.x) + 1u;   // >= 1
  const int msb = 31 - __clz(x);
  const int frac = msb >= 2 ? (int)((x >> (msb - 2)) & 3u) : (int)((x << (2 - msb)) & 3u);
  return kOrderBins - 1 - min(kOrderBins - 1, 4 * msb + frac);  // longest first
}

__global__ void __launch_bounds__(kOrderThreads)
    k_tile_order(const int2* __restrict__ ranges, int tiles, int32_t* __restrict__ order) {
  pdl_wait();
  __shared__ int cnt[kOrderBins];
  if (threadIdx.x < kOrderBins) cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int t = threadIdx.x; t < tiles; t += kOrderThreads) atomicAdd(&cnt[order_bin(ranges[t])], 1);
  __syncthreads();
  if (threadIdx.x < 32) {  // exclusive scan of the bins, 4 per lane
    const int lane = threadIdx.x;
    int v[kOrderBins / 32], sum = 0;
#pragma unroll
    for (int k = 0; k < kOrderBins / 32; ++k) {
      v[k] = cnt[lane * (kOrderBins / 32) + k];
      sum += v[k];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    int run = incl - sum;
#pragma unroll
    for (int k = 0; k < kOrderBins / 32; ++k) {
      cnt[lane * (kOrderBins / 32) + k] = run;
      run += v[k];
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < tiles; t += kOrderThreads)
    order[atomicAdd(&cnt[order_bin(ranges[t])], 1)] = t;
}

int launch_tile_order(const int2* ranges, int tiles, int32_t* order, cudaStream_t st) {
  launch_pdl(k_tile_order, dim3(1), dim3(kOrderThreads), 0, st, ranges, tiles, order);
  return check_launch("tile order");
}

// ------------------------------------------------------------- forward
// A block's staged batch: the records' float4s vector-major (rec[v * kBatch +
// slot]: v0, v1 and the further channels), so the per-slot reads of a warp's
// walk are broadcasts, and each record's mask of warps.
template <int K>
struct DrawBatch {
  static constexpr int V = RecordLayout<K>::kVec4;
  float4 rec[(V - 1) * kBatch];
  uint8_t mask[kBatch];

  __device__ __forceinline__ void channels(int j, float v1w, float* f) const {
    f[0] = v1w;  // channel 0 sits in v1.w
#pragma unroll
    for (int k = 1; k < K; ++k) {
      const float4 q = rec[(2 + (k - 1) / 4) * kBatch + j];
      f[k] = ((k - 1) & 3) == 0 ? q.x : ((k - 1) & 3) == 1 ? q.y : ((k - 1) & 3) == 2 ? q.z : q.w;
    }
  }
};

// Composites one 16x16 tile of one image (draw_weight / draw_color,
// gsplatcu/kernel.cu:283-372): ranges/gsid/records of that image's tile
// lists, K channels, final_tau of empty tiles = tau_init.  Called by all
// threads of a block; it starts with a block barrier, so the buffer may still
// be in use by the block's previous tile when it is called.
template <int K>
__device__ __forceinline__ void draw_tile(int tile, int H, int W, int gx,
                                          const int2* __restrict__ ranges,
                                          const int32_t* __restrict__ gsid,
                                          const float4* __restrict__ records, float tau_init,
                                          float* __restrict__ out, int32_t* __restrict__ contrib,
                                          float* __restrict__ final_tau, DrawBatch<K>& b) {
  constexpr int V = RecordLayout<K>::kVec4;
  const int X0 = (tile % gx) * kTile, Y0 = (tile / gx) * kTile;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int px = X0 + (w & 1) * 8 + (lane & 7), py = Y0 + (w >> 1) * 4 + (lane >> 3);
  const bool inside = px < W && py < H;
  const int2 rg = ranges[tile];
  const int n = rg.y - rg.x;
  float acc[K];
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = 0.f;
  float T = 1.f;
  int cont = 0;
  bool done = !inside;
  for (int base = 0; base < n; base += kBatch) {
    const int cnt = min(kBatch, n - base);
    __syncthreads();
    if ((int)threadIdx.x < cnt) {
      const float4* src = records + (int64_t)gsid[rg.x + base + threadIdx.x] * V;
      const float4 v0 = __ldg(src), v1 = __ldg(src + 1), v2 = __ldg(src + 2);
      b.rec[threadIdx.x] = v0;
      b.rec[kBatch + threadIdx.x] = v1;
#pragma unroll
      for (int v = 3; v < V; ++v) b.rec[(v - 1) * kBatch + threadIdx.x] = __ldg(src + v);
      b.mask[threadIdx.x] = (uint8_t)region_mask<2, 4, 8, 4>(v0, v1, v2, X0, Y0);
    }
    __syncthreads();
    if (!__all_sync(0xffffffffu, done)) {
      for (int s = 0; s < cnt; s += 32) {
        const int j = s + lane;
        unsigned mask = __ballot_sync(0xffffffffu, j < cnt && ((b.mask[j] >> w) & 1));
        while (mask) {
          const int jj = s + __ffs(mask) - 1;
          mask &= mask - 1;
          if (mask) {
            // two records at once: both opacity terms first, so that their
            // exp() chains overlap, then the two blends in list order
            const int jb = s + __ffs(mask) - 1;
            mask &= mask - 1;
            if (done) continue;
            const float4 a0 = b.rec[jj], a1 = b.rec[kBatch + jj];
            const float4 b0 = b.rec[jb], b1 = b.rec[kBatch + jb];
            const float pa = fminf(0.f, half_form(a0.z, a0.w, a1.x, a0.x - (float)px, a0.y - (float)py));
            const float pb = fminf(0.f, half_form(b0.z, b0.w, b1.x, b0.x - (float)px, b0.y - (float)py));
            const float apa = fminf(kAlphaMax, a1.z * expf(pa));
            const float apb = fminf(kAlphaMax, b1.z * expf(pb));
            if (pa >= a1.y) {
              float f[K];
              b.channels(jj, a1.w, f);
#pragma unroll
              for (int k = 0; k < K; ++k) acc[k] += T * apa * f[k];
              cont = base + jj + 1;
              T *= (1.f - apa);
              if (T < kTransMin) done = true;
            }
            if (!done && pb >= b1.y) {
              float f[K];
              b.channels(jb, b1.w, f);
#pragma unroll
              for (int k = 0; k < K; ++k) acc[k] += T * apb * f[k];
              cont = base + jb + 1;
              T *= (1.f - apb);
              if (T < kTransMin) done = true;
            }
            continue;
          }
          if (done) continue;
          const float4 v0 = b.rec[jj];           // ux uy, conic a b
          const float4 v1 = b.rec[kBatch + jj];  // conic c, threshold, alpha, ch0
          const float p = fminf(0.f, half_form(v0.z, v0.w, v1.x, v0.x - (float)px, v0.y - (float)py));
          if (!(p >= v1.y)) continue;
          const float ap = fminf(kAlphaMax, v1.z * expf(p));
          float f[K];
          b.channels(jj, v1.w, f);
#pragma unroll
          for (int k = 0; k < K; ++k) acc[k] += T * ap * f[k];
          cont = base + jj + 1;
          T *= (1.f - ap);
          if (T < kTransMin) done = true;
        }
        if (__all_sync(0xffffffffu, done)) break;
      }
    }
    if (!__syncthreads_or(!done)) break;
  }
  if (inside) {
    const int64_t pix = (int64_t)py * W + px, hw = (int64_t)H * W;
#pragma unroll
    for (int k = 0; k < K; ++k) out[k * hw + pix] = acc[k];
    contrib[pix] = cont;
    final_tau[pix] = n > 0 ? T : tau_init;
  }
}

template <int K>
__global__ void __launch_bounds__(kDrawThreads, 4)
    k_draw(int H, int W, int gx, const int2* __restrict__ ranges, const int32_t* __restrict__ gsid,
           const float4* __restrict__ records, const int32_t* __restrict__ order,
           float tau_init, float* __restrict__ out, int32_t* __restrict__ contrib,
           float* __restrict__ final_tau) {
  pdl_wait();
  __shared__ DrawBatch<K> batch;
  draw_tile<K>(order[blockIdx.x], H, W, gx, ranges, gsid, records, tau_init, out, contrib,
               final_tau, batch);
}

// ------------------------------------------------- batched (persistent) draw
// One image of a batch: its packed records, tile lists and outputs, and the
// index of its first tile in the batch's work queue.
struct DrawJob {
  const float4* records;
  const int2* ranges;
  const int32_t* gsid;
  float* out;
  int32_t* contrib;
  float* final_tau;
  int W, H, gx, item0;
  float tau_init;
  int pad[3];
};
static_assert(sizeof(DrawJob) == 80, "DrawJob layout");

// Device work queue of a batch: (image, tile) items numbered 0..total-1
// image by image; `next` is the next unclaimed item (zero at launch).
struct DrawQueue {
  uint32_t njobs, total, next, pad;
  DrawJob jobs[1];  // njobs entries
};

// Persistent compositing of a batch of images (the palette-edit renders of
// several requests): a grid of a few blocks per SM, each block claims the
// next (image, tile) item with one atomic add, composites that tile exactly
// as k_draw does, and claims again until the queue is empty.  The tiles of
// large and small images share the SMs, whatever the images' sizes.
template <int K>
__global__ void __launch_bounds__(kDrawThreads, 4) k_draw_queue(DrawQueue* __restrict__ q) {
  pdl_wait();
  __shared__ DrawBatch<K> batch;
  __shared__ int s_item, s_job;
  const int total = (int)q->total, njobs = (int)q->njobs;
  for (;;) {
    if (threadIdx.x == 0) {
      const int item = (int)atomicAdd(&q->next, 1u);
      int j = 0;
      while (j + 1 < njobs && (int)q->jobs[j + 1].item0 <= item) ++j;
      s_item = item;
      s_job = j;
    }
    __syncthreads();
    const int item = s_item;
    if (item >= total) break;
    const DrawJob& jb = q->jobs[s_job];
    draw_tile<K>(item - jb.item0, jb.H, jb.W, jb.gx, jb.ranges, jb.gsid, jb.records, jb.tau_init,
                 jb.out, jb.contrib, jb.final_tau, batch);
    __syncthreads();  // s_item / s_job are rewritten by the next claim
  }
}

size_t draw_queue_bytes(int max_jobs) {
  return offsetof(DrawQueue, jobs) + (size_t)(max_jobs > 0 ? max_jobs : 1) * sizeof(DrawJob);
}

// Host side: the queue image the caller copies to the device.
int draw_queue_pack(const DrawJobDesc* jobs, int njobs, void* host_table, size_t table_bytes) {
  if (draw_queue_bytes(njobs) > table_bytes) return GSB_ERR_CAPACITY;
  DrawQueue* q = (DrawQueue*)host_table;
  uint32_t item = 0;
  for (int i = 0; i < njobs; ++i) {
    const DrawJobDesc& d = jobs[i];
    const SplatState s = carve_state((void*)d.state, d.n, d.channels, d.height, d.width);
    DrawJob& j = q->jobs[i];
    j.records = s.records;
    j.ranges = (const int2*)d.ranges;
    j.gsid = d.gsid;
    j.out = d.out;
    j.contrib = d.contrib;
    j.final_tau = d.final_tau;
    j.W = d.width;
    j.H = d.height;
    j.gx = div_up(d.width, kTile);
    j.item0 = (int)item;
    j.tau_init = d.tau_init;
    j.pad[0] = j.pad[1] = j.pad[2] = 0;
    item += (uint32_t)(div_up(d.width, kTile) * div_up(d.height, kTile));
  }
  q->njobs = (uint32_t)njobs;
  q->total = item;
  q->next = 0;
  q->pad = 0;
  return GSB_OK;
}

int launch_draw_queue(int channels, const void* dev_table, int grid, cudaStream_t st) {
  DrawQueue* q = (DrawQueue*)dev_table;
  switch (channels) {
#define GSB_K(KK)                                                                          \
  case KK:                                                                                 \
    launch_pdl(k_draw_queue<KK>, dim3(grid), dim3(kDrawThreads), 0, st, q);             \
    break;
    GSB_K(1) GSB_K(2) GSB_K(3) GSB_K(4) GSB_K(5) GSB_K(6) GSB_K(7) GSB_K(8)
#undef GSB_K
    default: return GSB_ERR_INVALID_ARGUMENT;
  }
  return check_launch("draw_queue");
}

// ------------------------------------------------------------ launchers
int launch_draw(int64_t n, int H, int W, int channels, const int32_t* ranges, const int32_t* gsid,
                const SplatState& s, float tau_init, float* out, int32_t* contrib,
                float* final_tau, cudaStream_t st) {
  (void)n;
  const int gx = div_up(W, kTile), gy = div_up(H, kTile);
  const int tiles = gx * gy;
  if (tiles == 0) return GSB_OK;
  const int2* rg = (const int2*)ranges;
  if (channels < 1 || channels > 8) return GSB_ERR_INVALID_ARGUMENT;
  const int rc = launch_tile_order(rg, tiles, s.tile_order, st);
  if (rc) return rc;
  switch (channels) {
#define GSB_K(KK)                                                                           \
  case KK:                                                                                  \
    launch_pdl(k_draw<KK>, dim3(tiles), dim3(kDrawThreads), 0, st, H, W, gx, rg, gsid,       \
               (const float4*)s.records, (const int32_t*)s.tile_order, tau_init, out, contrib,   \
               final_tau);                                                                      \
    break;
    GSB_K(1) GSB_K(2) GSB_K(3) GSB_K(4) GSB_K(5) GSB_K(6) GSB_K(7) GSB_K(8)
#undef GSB_K
    default: return GSB_ERR_INVALID_ARGUMENT;
  }
  return check_launch("splat_draw");
}

}  // namespace gsb
