// Tile lists without sorting patches: the Gaussians are sorted by depth key, then
// every tile's list is filled in that order.
//
// The tile lists are ordered by (depth key, Gaussian index) within each tile
// (see binning.cu).  Instead of sorting one (tile, depth) key per patch -- 3 or 4
// radix passes over every patch -- this path
//   1. sorts the Gaussians that have patches by depth key (stable, 1 or 2 passes
//      over at most N elements) and gathers their rectangles in that order;
//   2. cuts the sequence into chunks of about equal patches, counts each chunk's
//      patches per tile (a 2-D difference array: four adds per Gaussian) and
//      scans the counts, over the chunks per tile and over the tiles (which are
//      the ranges);
//   3. expands each chunk and writes every patch at its tile's cursor, in order;
//      each warp owns a part of the chunk and a cursor per tile.
// No key is written, and each patch is expanded and stored once.
//
// What bounds it: step 3, by issue rate and by the scattered 4-byte stores (a
// patch's neighbours in memory belong to other chunks, so a store writes a 32-byte
// sector of its own when its tile's list is short).  A chunk is one block per SM
// and band because each needs counters for the band's tiles; more chunks shorten
// the serial part but multiply the counts (chunks x tiles words) that step 2 scans.
// All steps together: 1M Gaussians, 3.3M patches, 1080p, 0.128 ms
// (radix over patches: 0.169), of which the fill takes 0.054; 3M, 20.8M patches,
// 4K, 0.56 ms (1.11), fill 0.36.  Every band reads its chunk's Gaussians, so an image
// of many bands needs many patches per Gaussian to gain (the rule is in capi.cu).
#include <algorithm>

#include "gsb_common.cuh"
#include "gsb_internal.h"
#include "gsb_radix.cuh"

namespace gsb {

constexpr int kListThreads = 256, kListWarps = kListThreads / 32;
constexpr int kGroupSize = 256;     // Gaussians per unit of the chunk split
constexpr int kBandCells = 3072;    // cells a block keeps counters for (3 blocks per SM)
constexpr int kCountThreads = 512;
constexpr int kCountCells = 48 * 1024;  // cells of a counting block (192 KB)
constexpr int kRowGroup = 4;        // tile rows dealt to the bands at a time
constexpr int kSplitWeight = 4;     // weight of a Gaussian besides its patches
constexpr int kMaxChunks = 148;     // one block per SM and band; sizes are asked for without a device

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Dynamic shared memory limits of the kernels: the same for every image, since the
// attribute belongs to the function and host threads render different sizes at the
// same time.  A band of the fill has at most kBandCells cells and rows of at most
// kMaxPitch.
constexpr int kMaxPitch = kBandCells / kRowGroup;
constexpr int kCountSmemMax = kCountCells * 4;
constexpr int kFillSmemMax = (kBandCells + kListWarps * (kBandCells + kMaxPitch) / 2) * 4;
constexpr int kSortSmem = kSortTile * 8 + (8 * kRadixBins + 2 * kRadixBins + 8) * 4;

static int bits_of(uint32_t v) { return v ? 32 - __builtin_clz(v) : 0; }

// Tile rows are dealt to the bands in groups of kRowGroup, so that the bands of
// an image carry about equal loads and a Gaussian rarely meets more than two.  A
// band numbers its rows consecutively, and a run of image rows is a run of band
// rows: `below` counts the band's rows among the image's rows [0, r), r < 2^16.
struct BandRows {
  int band, period;     // period = kRowGroup * bands
  uint32_t inv_period;  // ceil(2^32 / period): exact quotients for r * period < 2^32
  __host__ __device__ BandRows(int band_, int bands)
      : band(band_), period(kRowGroup * bands),
        inv_period((uint32_t)(((uint64_t(1) << 32) + period - 1) / period)) {}
  __device__ BandRows(int band_, int bands, uint32_t inv)
      : band(band_), period(kRowGroup * bands), inv_period(inv) {}
  __host__ __device__ __forceinline__ int below(int r) const {
    const int q = (int)(((uint64_t)(uint32_t)r * inv_period) >> 32);
    const int in = r - q * period - kRowGroup * band;
    return q * kRowGroup + (in < 0 ? 0 : in > kRowGroup ? kRowGroup : in);
  }
};

// Dynamic shared memory of an image's counting and filling blocks.
static size_t count_bytes(const ListPlan& p) { return (size_t)(p.count_rows + 1) * (p.gx + 1) * 4; }
static size_t fill_bytes(const ListPlan& p) {
  return (size_t)(p.band_rows * p.pitch + kListWarps * ((p.band_rows + 1) * p.pitch / 2)) * 4;
}

ListPlan make_list_plan(int64_t n, int H, int W, int64_t M, uint32_t max_dkey) {
  ListPlan p{};
  p.gx = div_up(W, kTile);
  p.gy = div_up(H, kTile);
  p.tiles = (int64_t)p.gx * p.gy;
  p.n = n;
  p.M = M;
  p.dkey_bits = bits_of(max_dkey);
  p.ok = n > 0 && n < (int64_t(1) << 30) && M > 0 && p.tiles > 0 &&
         (p.gx + 4) * kRowGroup <= kBandCells && p.gy < 16384;
  if (!p.ok) return p;
  p.passes = std::max(1, (p.dkey_bits + kRadixBits - 1) / kRadixBits);
  p.digit_bits = std::max(1, (p.dkey_bits + p.passes - 1) / p.passes);
  // a chunk's Gaussians (at most its weight / (kSplitWeight + 1) and one group)
  // fit the 16-bit counters; few patches need few chunks
  const int64_t weight = M + kSplitWeight * n;
  p.chunks = (int)std::min<int64_t>(kMaxChunks, (M + 4095) / 4096);
  p.chunks = (int)std::max<int64_t>(p.chunks, weight / ((kSplitWeight + 1) * 60000) + 1);
  p.pitch = (p.gx + 2) & ~1;  // cells per row: two per word, an odd number of words
  p.pitch += p.pitch / 2 % 2 ? 0 : 2;
  const int groups = (p.gy + kRowGroup - 1) / kRowGroup;
  p.bands = div_up(groups, kBandCells / (p.pitch * kRowGroup));
  p.band_rows = BandRows(0, p.bands).below(p.gy);  // of the largest
  p.count_bands = div_up((p.gy + 1) * (int64_t)(p.gx + 1), kCountCells);
  while (p.count_bands > 1 &&
         (BandRows(0, p.count_bands).below(p.gy) + 1) * (p.gx + 1) > kCountCells)
    ++p.count_bands;
  p.count_rows = BandRows(0, p.count_bands).below(p.gy);
  p.ok = count_bytes(p) <= kCountSmemMax && fill_bytes(p) <= kFillSmemMax;  // (every image's)
  p.sort_blocks = (n + kSortTile - 1) / kSortTile;
  p.groups = (n + kGroupSize - 1) / kGroupSize;
  size_t off = 0;
  const auto take = [&off](size_t bytes) {
    const size_t at = off;
    off += align256(bytes);
    return at;
  };
  p.off_keys[0] = take((size_t)n * 4);
  p.off_keys[1] = take((size_t)n * 4);
  p.off_vals[0] = take((size_t)n * 4);
  p.off_vals[1] = take((size_t)n * 4);
  p.off_rects = take((size_t)n * 8);
  p.off_hist = take((size_t)kRadixBins * p.sort_blocks * 4);
  p.off_digit_tot = take((size_t)kRadixBins * 4);
  p.off_groups = take((size_t)p.groups * 4);
  p.off_bounds = take((size_t)(p.chunks + 1) * 4 + 4);  // chunk bounds, then the visible count
  p.off_counts = take((size_t)p.chunks * p.tiles * 4);
  p.off_tile_tot = take((size_t)p.tiles * 4);
  p.bytes_total = off;
  return p;
}

// Rectangles of the depth-sorted Gaussians, and each group's weight.
__global__ void __launch_bounds__(kGroupSize)
    k_sorted_rects(const uint32_t* __restrict__ visible, const int32_t* __restrict__ ids,
                   const uint2* __restrict__ rects, uint2* __restrict__ sorted,
                   uint32_t* __restrict__ groups) {
  pdl_wait();
  __shared__ uint32_t warp_tot[8];
  const int64_t i = (int64_t)blockIdx.x * kGroupSize + threadIdx.x;
  uint32_t weight = 0;
  if (i < (int64_t)*visible) {
    const uint2 r = rects[ids[i]];
    sorted[i] = r;
    weight = ((r.y & 0xffffu) - (r.x & 0xffffu)) * ((r.y >> 16) - (r.x >> 16)) + kSplitWeight;
  }
  uint32_t tot;
  block_excl_scan256(weight, warp_tot, &tot);
  if (threadIdx.x == 0) groups[blockIdx.x] = tot;
}

// Sum of v[0, n) over the block's 256 threads.
__device__ __forceinline__ unsigned long long block_sum256(const uint32_t* __restrict__ v, int n,
                                                           unsigned long long* warp_tot) {
  unsigned long long t = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += 256) t += v[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = t;
  __syncthreads();
  t = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) t += warp_tot[k];
  __syncthreads();
  return t;
}

// Chunk b starts at the first group whose preceding weight is at least b /
// chunks of the total.  Each block places the chunks that start in its 256
// groups; the sums before them it forms itself.
__global__ void __launch_bounds__(256)
    k_chunk_bounds(const uint32_t* __restrict__ groups, int n_groups, int chunks,
                   uint32_t* __restrict__ bounds) {
  pdl_wait();
  __shared__ unsigned long long wide[8];
  __shared__ uint32_t warp_tot[8];
  const int first = blockIdx.x * 256, g = first + threadIdx.x;
  const unsigned long long before_block = block_sum256(groups, first, wide);
  const unsigned long long total =
      before_block + block_sum256(groups + first, n_groups - first, wide);
  if (total == 0ull) {
    for (int b = threadIdx.x; blockIdx.x == 0 && b <= chunks; b += 256) bounds[b] = 0u;
    return;
  }
  const uint32_t mine = g < n_groups ? groups[g] : 0u;
  const unsigned long long before = before_block + block_excl_scan256(mine, warp_tot, nullptr);
  if (g >= n_groups) return;
  // the chunks b with prefix(g - 1) * chunks < b * total <= prefix(g) * chunks
  // start at g; what follows the last group starts past it
  const int last = (int)(before * chunks / total);
  const int start = g == 0 ? 0 : (int)((before - groups[g - 1]) * chunks / total) + 1;
  for (int b = start; b <= last; ++b) bounds[b] = (uint32_t)g;
  if (g == n_groups - 1)
    for (int b = last + 1; b <= chunks; ++b) bounds[b] = (uint32_t)n_groups;
}

// The Gaussians [first, last) of a chunk, and a band.
struct ListWork {
  int64_t first, last;
  BandRows rows;
  int count;  // rows of the band
};
__device__ __forceinline__ int image_row(int y, const ListWork& k) {
  return y / kRowGroup * k.rows.period + k.rows.band * kRowGroup + y % kRowGroup;
}
__device__ __forceinline__ ListWork list_work(const uint32_t* bounds, const uint32_t* visible,
                                              int gy, uint32_t inv_period) {
  ListWork k{0, 0, BandRows((int)blockIdx.y, (int)gridDim.y, inv_period), 0};
  const int64_t v = *visible;
  k.first = min(v, (int64_t)bounds[blockIdx.x] * kGroupSize);
  k.last = min(v, (int64_t)bounds[blockIdx.x + 1] * kGroupSize);
  k.count = k.rows.below(gy);
  return k;
}

// Patches per tile of one chunk in one band: four adds per Gaussian into a
// difference array, then running sums along its rows and columns.
__global__ void __launch_bounds__(kCountThreads)
    k_tile_counts(const uint2* __restrict__ rects, const uint32_t* __restrict__ bounds,
                  const uint32_t* __restrict__ visible, int gx, int gy, uint32_t inv_period,
                  uint32_t* __restrict__ counts) {
  pdl_wait();
  extern __shared__ int32_t diff[];  // [rows + 1][gx + 1]
  const ListWork k = list_work(bounds, visible, gy, inv_period);
  const int rows = k.count, pitch = gx + 1;
  for (int t = threadIdx.x; t < (rows + 1) * pitch; t += kCountThreads) diff[t] = 0;
  __syncthreads();
  for (int64_t i = k.first + threadIdx.x; i < k.last; i += kCountThreads) {
    const uint2 r = rects[i];
    const int x0 = r.x & 0xffffu, x1 = r.y & 0xffffu;
    const int y0 = k.rows.below(r.x >> 16);
    const int y1 = k.rows.below(r.y >> 16);
    if (y0 < y1) {
      atomicAdd(&diff[y0 * pitch + x0], 1);
      atomicAdd(&diff[y0 * pitch + x1], -1);
      atomicAdd(&diff[y1 * pitch + x0], -1);
      atomicAdd(&diff[y1 * pitch + x1], 1);
    }
  }
  __syncthreads();
  // columns first (thread per column: conflict-free), then rows by warps
  for (int x = threadIdx.x; x < gx; x += kCountThreads) {
    int run = 0;
    for (int y = 0; y < rows; ++y) {
      run += diff[y * pitch + x];
      diff[y * pitch + x] = run;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t* out = counts + (int64_t)blockIdx.x * gx * gy;
  for (int y = threadIdx.x >> 5; y < rows; y += (kCountThreads / 32)) {
    int carry = 0;
    for (int x = lane; x - lane < gx; x += 32) {
      int v = x < gx ? diff[y * pitch + x] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
      }
      v += carry;
      if (x < gx) out[(int64_t)image_row(y, k) * gx + x] = (uint32_t)v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
}

// Per tile: exclusive sums over the chunks, and the tile's total.
__global__ void __launch_bounds__(64)
    k_chunk_prefix(uint32_t* __restrict__ counts, int64_t tiles, int chunks,
                   uint32_t* __restrict__ tile_tot) {
  pdl_wait();
  const int64_t t = (int64_t)blockIdx.x * 64 + threadIdx.x;
  if (t >= tiles) return;
  uint32_t run = 0;
  constexpr int kAhead = 16;
  for (int c0 = 0; c0 < chunks; c0 += kAhead) {
    uint32_t v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      v[u] = c0 + u < chunks ? counts[(int64_t)(c0 + u) * tiles + t] : 0u;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (c0 + u < chunks) counts[(int64_t)(c0 + u) * tiles + t] = run;
      run += v[u];
    }
  }
  tile_tot[t] = run;
}

// Ranges: exclusive sums of the tile totals, each block forming the sum before
// its 256 tiles itself.  As getRanges leaves them (gsplatcu/kernel.cu:165-187):
// empty tiles are (0, 0), and so is the only tile of a single patch.  On a
// capacity overflow every range is empty.
__global__ void __launch_bounds__(256)
    k_tile_ranges(const uint32_t* __restrict__ tile_tot, int tiles, int64_t M, int dkey_bits,
                  const uint32_t* __restrict__ mdev, int2* __restrict__ ranges) {
  pdl_wait();
  __shared__ unsigned long long wide[8];
  __shared__ uint32_t warp_tot[8];
  const int first = blockIdx.x * 256, t = first + threadIdx.x;
  const uint32_t before_block = (uint32_t)block_sum256(tile_tot, first, wide);
  const uint32_t v = t < tiles ? tile_tot[t] : 0u;
  uint32_t here;
  const uint32_t before = before_block + block_excl_scan256(v, warp_tot, &here);
  bool none = capacity_overflow(M, mdev, dkey_bits);
  if (before_block + here == 1u)  // (uniform) the only patch?
    none |= block_sum256(tile_tot + first, tiles - first, wide) + before_block == 1ull;
  if (t < tiles)
    ranges[t] = none || v == 0u ? make_int2(0, 0) : make_int2((int)before, (int)(before + v));
}

// A warp's queue of Gaussians that meet the band: their rectangles in band rows
// and indices, in order.  Filled 32 candidates at a time and expanded 32 entries
// at a time, so the expansion runs on full warps whatever part of the candidates
// lies in the band.
struct WarpQueue {
  uint2 rect[64];  // x0 | y0 << 16, width | height << 16
  int32_t id[64];
};

// Expands the first `n` (<= 32) queue entries: lanes take their patches in order,
// 32 at a time, and call f(cell in the band, entry, valid) with all lanes.  A
// window's entries are found from the starts that fall into it (one reduction).
template <typename F>
__device__ __forceinline__ void expand_queue(WarpQueue& q, int n, int pitch, F f) {
  const int lane = threadIdx.x & 31;
  uint32_t c = 0;
  float inv_w = 0.f;
  if (lane < n) {
    const uint32_t wh = q.rect[lane].y;
    c = (wh & 0xffffu) * (wh >> 16);
    inv_w = __fdividef(1.f, (float)(wh & 0xffffu));
  }
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t start = incl - c;  // of this lane's entry
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  int begun = 0;  // entries that start before the window
  for (uint32_t p0 = 0; p0 < total; p0 += 32) {
    const uint32_t at = start - p0;
    const unsigned starts =
        __reduce_or_sync(0xffffffffu, lane < n && at < 32u ? 1u << at : 0u);
    const bool ok = p0 + lane < total;
    // (every valid lane has an entry that starts at or before it)
    const int L = ok ? begun + __popc(starts & (0xffffffffu >> (31 - lane))) - 1 : 0;
    begun += __popc(starts);
    const uint32_t local = p0 + lane - __shfl_sync(0xffffffffu, start, L);
    const float iw = __shfl_sync(0xffffffffu, inv_w, L);
    const uint2 r = q.rect[L];
    // exact: (local + 1/2) / w is at least 1 / (2 w) from a whole number, far more
    // than the rounding of a quotient below 2^12
    const uint32_t ty = (uint32_t)(((float)local + 0.5f) * iw);
    const int cell = (int)(((r.x >> 16) + ty) * pitch + (r.x & 0xffffu) + (local - ty * (r.y & 0xffffu)));
    f(ok ? cell : 0, L, ok);
  }
  __syncwarp();  // the queue may be rewritten
}

// Runs a warp's Gaussians [g0, g1) through the queue.
template <typename F>
__device__ __forceinline__ void expand_range(WarpQueue& q, const uint2* __restrict__ rects,
                                             const int32_t* __restrict__ ids, int64_t g0,
                                             int64_t g1, const ListWork& k, int pitch, F f) {
  const int lane = threadIdx.x & 31;
  constexpr int kAhead = 4;  // candidates per lane in flight during the expansion
  int n = 0;
  uint2 next[kAhead];
  int32_t next_id[kAhead];
  const auto fetch = [&](int64_t base) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t i = base + 32 * u + lane;
      next[u] = i < g1 ? rects[i] : make_uint2(0u, 0u);  // (an empty rectangle)
      next_id[u] = i < g1 ? ids[i] : 0;
    }
  };
  fetch(g0);
  uint2 cur[kAhead];
  int32_t cur_id[kAhead];
  int u = kAhead;
  for (int64_t i = g0; i < g1; i += 32, ++u) {
    if (u == kAhead) {
#pragma unroll
      for (int v = 0; v < kAhead; ++v) {
        cur[v] = next[v];
        cur_id[v] = next_id[v];
      }
      fetch(i + 32 * kAhead);
      u = 0;
    }
    const uint2 r = cur[0];
    const int32_t me = cur_id[0];
#pragma unroll
    for (int v = 0; v + 1 < kAhead; ++v) {
      cur[v] = cur[v + 1];
      cur_id[v] = cur_id[v + 1];
    }
    const int x0 = r.x & 0xffffu, x1 = r.y & 0xffffu;
    const int y0 = k.rows.below(r.x >> 16), y1 = k.rows.below(r.y >> 16);
    const bool in = y0 < y1 && x0 < x1;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (in) {
      const int at = n + __popc(m & ((1u << lane) - 1u));
      q.rect[at] = make_uint2((uint32_t)(x0 | (y0 << 16)),
                              (uint32_t)((x1 - x0) | ((y1 - y0) << 16)));
      q.id[at] = me;
    }
    n += __popc(m);
    __syncwarp();
    if (n >= 32) {
      expand_queue(q, 32, pitch, f);
      n -= 32;
      uint2 rest = make_uint2(0u, 0u);
      int32_t rid = 0;
      if (lane < n) {
        rest = q.rect[32 + lane];
        rid = q.id[32 + lane];
      }
      __syncwarp();
      if (lane < n) {
        q.rect[lane] = rest;
        q.id[lane] = rid;
      }
      __syncwarp();
    }
  }
  if (n) expand_queue(q, n, pitch, f);
}

// Patches per tile of a warp's Gaussians [g0, g1), two 16-bit cells per word: a
// difference array as in k_tile_counts (a cell's sum stays within 16 bits, but
// its borrow reaches the other half of the word until the two are separated),
// running sums along the columns, then along the rows.  Cheaper than expanding
// the patches a second time: 4 adds per Gaussian and 20 operations per word.
__device__ __forceinline__ void warp_counts(uint32_t* cells, const uint2* __restrict__ rects,
                                            int64_t g0, int64_t g1, const ListWork& k, int pitch) {
  const int lane = threadIdx.x & 31, pw = pitch / 2;
  const auto add = [cells, pitch](int y, int x, uint32_t v) {
    atomicAdd(&cells[(y * pitch + x) >> 1], x & 1 ? v << 16 : v);
  };
  for (int t = lane; t < (k.count + 1) * pw; t += 32) cells[t] = 0u;
  __syncwarp();
  constexpr int kAhead = 8;
  for (int64_t i0 = g0 + lane; i0 - lane < g1; i0 += 32 * kAhead) {
    uint2 r[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t i = i0 + 32 * u;
      r[u] = i < g1 ? rects[i] : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int x0 = r[u].x & 0xffffu, x1 = r[u].y & 0xffffu;
      const int y0 = k.rows.below(r[u].x >> 16), y1 = k.rows.below(r[u].y >> 16);
      if (y0 < y1) {
        add(y0, x0, 1u);
        add(y0, x1, ~0u);
        add(y1, x0, ~0u);
        add(y1, x1, 1u);
      }
    }
  }
  __syncwarp();
  for (int c = lane; c < pw; c += 32) {
    int lo = 0, hi = 0;
    for (int y = 0; y < k.count; ++y) {
      const uint32_t v = cells[y * pw + c];
      const int d = (int16_t)(v & 0xffffu);
      lo += d;
      hi += (int)(v - (uint32_t)d) >> 16;
      cells[y * pw + c] = (uint32_t)(lo & 0xffff) | ((uint32_t)hi << 16);
    }
  }
  __syncwarp();
  for (int y = lane; y < k.count; y += 32) {
    int run = 0;
    for (int c = 0; c < pw; ++c) {
      const uint32_t v = cells[y * pw + c];
      run += (int16_t)(v & 0xffffu);
      const int first = run;
      run += (int16_t)(v >> 16);
      cells[y * pw + c] = (uint32_t)(first & 0xffff) | ((uint32_t)run << 16);
    }
  }
  __syncwarp();
}

// Writes one chunk's patches of one band into the tile lists.  Each warp takes
// a contiguous part of the chunk's Gaussians and counts its patches per tile;
// the counts become exclusive over the warps, and the patches are expanded and
// written at cursor[warp][tile] past the tile's start for this chunk.
__global__ void __launch_bounds__(kListThreads)
    k_tile_scatter(const uint2* __restrict__ rects, const int32_t* __restrict__ ids,
                   const uint32_t* __restrict__ bounds, const uint32_t* __restrict__ visible,
                   int gx, int gy, int pitch, uint32_t inv_period,
                   const uint32_t* __restrict__ counts, const int2* __restrict__ ranges, int64_t M,
                   int dkey_bits, const uint32_t* __restrict__ mdev, int32_t* __restrict__ out) {
  pdl_wait();
  if (capacity_overflow(M, mdev, dkey_bits)) return;
  extern __shared__ uint32_t list_smem[];
  __shared__ WarpQueue queues[kListWarps];
  const ListWork k = list_work(bounds, visible, gy, inv_period);
  if (k.first >= k.last) return;
  const int starts = k.count * pitch, words = (k.count + 1) * pitch / 2;
  uint32_t* start = list_smem;             // [rows][pitch]: the tile's list past earlier chunks
  uint32_t* cursors = list_smem + starts;  // [warps][words]: 16 bits per cell
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* mine = cursors + w * words;
  for (int y = w; y < k.count; y += kListWarps) {
    const int64_t tile = (int64_t)image_row(y, k) * gx;
    const uint32_t* before = counts + (int64_t)blockIdx.x * gx * gy + tile;
    for (int x = lane; x < gx; x += 32) start[y * pitch + x] = (uint32_t)ranges[tile + x].x + before[x];
  }
  const int64_t len = k.last - k.first;
  const int64_t g0 = k.first + len * w / kListWarps, g1 = k.first + len * (w + 1) / kListWarps;
  warp_counts(mine, rects, g0, g1, k, pitch);
  __syncthreads();
  for (int t = threadIdx.x; t < starts / 2; t += kListThreads) {  // two tiles at a time
    uint32_t run = 0;
#pragma unroll
    for (int v = 0; v < kListWarps; ++v) {
      const uint32_t c = cursors[v * words + t];
      cursors[v * words + t] = run;
      run += c;
    }
  }
  __syncthreads();
  WarpQueue& q = queues[w];
  const unsigned lt = (1u << lane) - 1u;
  expand_range(q, rects, ids, g0, g1, k, pitch, [&](int t, int L, bool ok) {
    // every lane claims a place at its tile's cursor; only if two lanes share a
    // tile (the cursor moved by more than one) the places are dealt in lane order
    const int half = 16 * (t & 1);
    uint32_t before = 0, after = 1;
    if (ok) before = (atomicAdd(&mine[t >> 1], 1u << half) >> half) & 0xffffu;
    __syncwarp();
    if (ok) after = (mine[t >> 1] >> half) & 0xffffu;
    if (__any_sync(0xffffffffu, after - before != 1u)) {
      const unsigned peers = __match_any_sync(0xffffffffu, ok ? t : -1);
      before = after - __popc(peers) + __popc(peers & lt);
    }
    if (ok) {
      const int64_t at = (int64_t)start[t] + before;
      if (at < M) out[at] = q.id[L];
    }
  });
}

int launch_tile_lists(const ListPlan& p, const SplatState& s, void* ws, int32_t* gsid_out,
                      int32_t* ranges_out, const uint32_t* mdev, cudaStream_t st) {
  char* b = (char*)ws;
  uint32_t* keys[2] = {(uint32_t*)(b + p.off_keys[0]), (uint32_t*)(b + p.off_keys[1])};
  int32_t* vals[2] = {(int32_t*)(b + p.off_vals[0]), (int32_t*)(b + p.off_vals[1])};
  uint2* rects = (uint2*)(b + p.off_rects);
  uint32_t* hist = (uint32_t*)(b + p.off_hist);
  uint32_t* dtot = (uint32_t*)(b + p.off_digit_tot);
  uint32_t* groups = (uint32_t*)(b + p.off_groups);
  uint32_t* bounds = (uint32_t*)(b + p.off_bounds);
  uint32_t* visible = bounds + p.chunks + 1;
  uint32_t* counts = (uint32_t*)(b + p.off_counts);
  uint32_t* tile_tot = (uint32_t*)(b + p.off_tile_tot);
  const int nbk = (int)p.sort_blocks;
  const size_t count_smem = count_bytes(p), list_smem = fill_bytes(p);
  const auto limit = [](const void* kern, int bytes) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
           cudaSuccess;
  };
  if (!limit((const void*)k_radix_downsweep<uint32_t, kVisible>, kSortSmem) ||
      !limit((const void*)k_radix_downsweep<uint32_t, kDevice>, kSortSmem) ||
      !limit((const void*)k_tile_counts, kCountSmemMax) ||
      !limit((const void*)k_tile_scatter, kFillSmemMax))
    return check_launch("tile lists (shared memory attribute)", 0);
  // 1. depth order of the Gaussians that have patches
  int src = 0;
  for (int pass = 0; pass < p.passes; ++pass) {
    const int shift = p.digit_bits * pass;
    const int bits = std::max(1, std::min(p.digit_bits, p.dkey_bits - shift));
    const uint32_t mask = (1u << bits) - 1u;
    if (pass == 0) {
      launch_pdl(k_radix_upsweep<uint32_t, kVisible>, dim3(nbk), dim3(kSortThreads), 0, st,
                 (const uint32_t*)s.dkeys, p.n, shift, mask, hist, p.sort_blocks,
                 (const uint32_t*)nullptr, (const uint32_t*)s.counts);
      launch_pdl(k_radix_scan, dim3(mask + 1), dim3(256), 0, st, hist, p.sort_blocks, dtot);
      launch_pdl(k_radix_downsweep<uint32_t, kVisible>, dim3(nbk), dim3(kSortThreads), kSortSmem,
                 st, (const uint32_t*)s.dkeys, (const int32_t*)nullptr, keys[0], vals[0], p.n, shift,
                 mask, (const uint32_t*)hist, (const uint32_t*)dtot, p.sort_blocks,
                 (const uint32_t*)nullptr, (const uint32_t*)s.counts, visible);
    } else {
      launch_pdl(k_radix_upsweep<uint32_t, kDevice>, dim3(nbk), dim3(kSortThreads), 0, st,
                 (const uint32_t*)keys[src], p.n, shift, mask, hist, p.sort_blocks,
                 (const uint32_t*)visible, (const uint32_t*)nullptr);
      launch_pdl(k_radix_scan, dim3(mask + 1), dim3(256), 0, st, hist, p.sort_blocks, dtot);
      launch_pdl(k_radix_downsweep<uint32_t, kDevice>, dim3(nbk), dim3(kSortThreads), kSortSmem, st,
                 (const uint32_t*)keys[src], (const int32_t*)vals[src], keys[src ^ 1],
                 vals[src ^ 1], p.n, shift, mask, (const uint32_t*)hist, (const uint32_t*)dtot,
                 p.sort_blocks, (const uint32_t*)visible, (const uint32_t*)nullptr,
                 (uint32_t*)nullptr);
      src ^= 1;
    }
    const int rc = check_launch("tile lists (depth pass)", 3);
    if (rc) return rc;
  }
  const int32_t* ids = vals[src];
  // 2. chunks, counts, ranges
  launch_pdl(k_sorted_rects, dim3((unsigned)p.groups), dim3(kGroupSize), 0, st,
             (const uint32_t*)visible, ids, (const uint2*)s.rects, rects, groups);
  launch_pdl(k_chunk_bounds, dim3((unsigned)((p.groups + 255) / 256)), dim3(256), 0, st, (const uint32_t*)groups, (int)p.groups,
             p.chunks, bounds);
  launch_pdl(k_tile_counts, dim3(p.chunks, p.count_bands), dim3(kCountThreads), count_smem, st,
             (const uint2*)rects, (const uint32_t*)bounds, (const uint32_t*)visible, p.gx, p.gy,
             BandRows(0, p.count_bands).inv_period, counts);
  launch_pdl(k_chunk_prefix, dim3((unsigned)((p.tiles + 63) / 64)), dim3(64), 0, st, counts,
             p.tiles, p.chunks, tile_tot);
  launch_pdl(k_tile_ranges, dim3((unsigned)((p.tiles + 255) / 256)), dim3(256), 0, st, (const uint32_t*)tile_tot, (int)p.tiles,
             p.M, p.dkey_bits, mdev, (int2*)ranges_out);
  // 3. lists
  launch_pdl(k_tile_scatter, dim3(p.chunks, p.bands), dim3(kListThreads), list_smem, st,
             (const uint2*)rects, ids, (const uint32_t*)bounds, (const uint32_t*)visible, p.gx, p.gy,
             p.pitch, BandRows(0, p.bands).inv_period, (const uint32_t*)counts, (const int2*)ranges_out, p.M, p.dkey_bits, mdev,
             gsid_out);
  return check_launch("tile lists", 6);
}

}  // namespace gsb
