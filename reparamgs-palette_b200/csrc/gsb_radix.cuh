// Stable LSD radix passes (upsweep, digit scan, downsweep) shared by the patch
// sort (binning.cu) and the depth sort of the tile lists (tile_lists.cu).
#pragma once

#include "gsb_common.cuh"
#include "gsb_internal.h"

namespace gsb {

// --------------------------------------------------------- block helpers
// Exclusive scan of one value per thread over a 256-thread block.
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t* warp_tot,
                                                       uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  uint32_t base = 0, tot = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t t = warp_tot[k];
    base += (k < w) ? t : 0u;
    tot += t;
  }
  __syncthreads();
  if (total) *total = tot;
  return base + incl - v;
}

// Patch count the sort kernels work on.  `mdev` null: the host-known count
// M.  Otherwise (capacity path, no host read-back) M is a capacity and the
// true count is the device total in mdev (stats words 0 and 3); a count
// above the capacity, or a depth key wider than `dkey_bits`, is an overflow:
// the kernels then stay inside the capacity and k_ranges leaves every range
// empty, so nothing downstream reads the unsorted entries.
__device__ __forceinline__ int64_t device_patches(int64_t M, const uint32_t* mdev) {
  if (!mdev) return M;
  const uint64_t m = (uint64_t)mdev[0] | ((uint64_t)mdev[3] << 32);
  return m > (uint64_t)M ? M : (int64_t)m;
}
__device__ __forceinline__ bool capacity_overflow(int64_t M, const uint32_t* mdev, int dkey_bits) {
  if (!mdev) return false;
  const uint64_t m = (uint64_t)mdev[0] | ((uint64_t)mdev[3] << 32);
  return m > (uint64_t)M || (dkey_bits < 32 && (mdev[1] >> dkey_bits) != 0u);
}

// ------------------------------------------------------------ radix sort
constexpr int kSortThreads = 256;
constexpr int kSortItems = 12;  // measured: 8 -> 12 keys per thread, 7 % less sort time
constexpr int kSortTile = kSortThreads * kSortItems;  // keys per block

// What a pass sorts: patches (M, or the device count under a capacity), the
// Gaussians that have patches (the first pass of the depth sort: M candidates,
// dropped where counts[i] is 0, values = indices), or as many elements as a
// device word says (its later passes).
enum SortSource { kPatches, kVisible, kDevice };

template <int SRC>
__device__ __forceinline__ int64_t sort_elements(int64_t M, const uint32_t* dev) {
  if (SRC == kPatches) return device_patches(M, dev);
  if (SRC == kDevice) return min(M, (int64_t)*dev);
  return M;
}

template <typename KT, int SRC>
__global__ void __launch_bounds__(kSortThreads)
    k_radix_upsweep(const KT* __restrict__ keys, int64_t M, int shift, uint32_t mask,
                    uint32_t* __restrict__ hist, int64_t nblocks, const uint32_t* __restrict__ mdev,
                    const uint32_t* __restrict__ counts) {
  pdl_wait();
  __shared__ uint32_t h[8][kRadixBins];
  M = sort_elements<SRC>(M, mdev);
  const int w = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < 8 * kRadixBins; k += kSortThreads) (&h[0][0])[k] = 0u;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile;
  // all of the thread's keys in flight before the histogram updates
  KT k[kSortItems];
  bool ok[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int64_t idx = base + r * kSortThreads + threadIdx.x;
    ok[r] = idx < M;
    k[r] = ok[r] ? keys[idx] : (KT)0;
    if (SRC == kVisible && ok[r]) ok[r] = counts[idx] > 0u;
  }
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    if (ok[r]) atomicAdd(&h[w][(uint32_t)(k[r] >> shift) & mask], 1u);
  }
  __syncthreads();
  for (uint32_t d = threadIdx.x; d <= mask; d += kSortThreads) {
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += h[k][d];
    hist[(int64_t)d * nblocks + blockIdx.x] = s;
  }
}

// One block per digit: exclusive scan of that digit's per-block counts.
static __global__ void __launch_bounds__(256)
    k_radix_scan(uint32_t* __restrict__ hist, int64_t nblocks, uint32_t* __restrict__ digit_tot) {
  pdl_wait();
  __shared__ uint32_t warp_tot[8];
  uint32_t* row = hist + (int64_t)blockIdx.x * nblocks;
  uint32_t carry = 0;
  constexpr int kItems = 8;  // consecutive counts per thread: one block scan per 2048
  for (int64_t base = 0; base < nblocks; base += 256 * kItems) {
    const int64_t j0 = base + (int64_t)threadIdx.x * kItems;
    uint32_t v[kItems], s = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      v[i] = j0 + i < nblocks ? row[j0 + i] : 0u;
      s += v[i];
    }
    uint32_t tot;
    uint32_t run = carry + block_excl_scan256(s, warp_tot, &tot);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (j0 + i < nblocks) row[j0 + i] = run;
      run += v[i];
    }
    carry += tot;
  }
  if (threadIdx.x == 0) digit_tot[blockIdx.x] = carry;
}

// Stable scatter of one digit pass.  Items of a block are ranked in their
// original order (warp w owns items [32 kSortItems w, 32 kSortItems (w+1)),
// lane-minor), staged in
// shared memory in digit order and written out in digit-contiguous runs.
// Thread t owns digits 2t and 2t+1 in the per-digit phases.
template <typename KT, int SRC>
__global__ void __launch_bounds__(kSortThreads)
    k_radix_downsweep(const KT* __restrict__ kin, const int32_t* __restrict__ vin,
                      KT* __restrict__ kout, int32_t* __restrict__ vout, int64_t M, int shift,
                      uint32_t mask, const uint32_t* __restrict__ hist,
                      const uint32_t* __restrict__ digit_tot, int64_t nblocks,
                      const uint32_t* __restrict__ mdev, const uint32_t* __restrict__ counts,
                      uint32_t* __restrict__ total_out) {
  pdl_wait();
  static_assert(kRadixBins == 2 * kSortThreads, "two digits per thread");
  M = sort_elements<SRC>(M, mdev);
  if ((int64_t)blockIdx.x * kSortTile >= M) return;  // whole block past the patches
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KT* sk = (KT*)smem_raw;
  int32_t* sv = (int32_t*)(sk + kSortTile);
  uint32_t* wcnt = (uint32_t*)(sv + kSortTile);  // [8][kRadixBins]
  uint32_t* lstart = wcnt + 8 * kRadixBins;      // [kRadixBins]
  uint32_t* gstart = lstart + kRadixBins;        // [kRadixBins]
  uint32_t* warp_tot = gstart + kRadixBins;      // [8]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int k = threadIdx.x; k < 8 * kRadixBins; k += kSortThreads) wcnt[k] = 0u;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kSortTile + w * (32 * kSortItems);
  KT key[kSortItems];
  int32_t val[kSortItems];
  uint32_t rnk[kSortItems], live = 0u;  // bit r: item r takes part
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int64_t idx = base + r * 32 + lane;
    const bool in = idx < M;
    key[r] = in ? kin[idx] : (KT)0;
    if (SRC == kVisible) {
      val[r] = (int32_t)idx;
      live |= (in && counts[idx] > 0u ? 1u : 0u) << r;
    } else {
      val[r] = in ? vin[idx] : 0;
      live |= (in ? 1u : 0u) << r;
    }
  }
  const uint32_t lt = (1u << lane) - 1u;
  const int nbits = 32 - __clz(mask);  // digit bits of this pass
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const bool ok = (live >> r) & 1u;
    const uint32_t d = ok ? ((uint32_t)(key[r] >> shift) & mask) : 0xffffu;
    // lanes with the same digit: one ballot per digit bit of this pass
    // (faster than __match_any_sync here: 0.181 -> 0.164 ms per sort of
    // 3.5M keys)
    uint32_t peers = __ballot_sync(0xffffffffu, ok);
    if (!ok) peers = ~peers;
    for (int b = 0; b < nbits; ++b) {
      const bool bit = (d >> b) & 1u;
      const uint32_t bm = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? bm : ~bm;
    }
    const uint32_t before = ok ? wcnt[w * kRadixBins + d] : 0u;
    rnk[r] = before + __popc(peers & lt);
    __syncwarp();
    if (ok && lane == __ffs(peers) - 1) wcnt[w * kRadixBins + d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive offsets across warps, block-local start, global start
  const uint32_t d0 = 2 * threadIdx.x, d1 = d0 + 1;
  uint32_t tot0 = 0, tot1 = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t c0 = wcnt[k * kRadixBins + d0], c1 = wcnt[k * kRadixBins + d1];
    wcnt[k * kRadixBins + d0] = tot0;
    wcnt[k * kRadixBins + d1] = tot1;
    tot0 += c0;
    tot1 += c1;
  }
  const uint32_t dt0 = d0 <= mask ? digit_tot[d0] : 0u, dt1 = d1 <= mask ? digit_tot[d1] : 0u;
  uint32_t cnt, all;  // elements of this block, of all blocks
  const uint32_t ls = block_excl_scan256(tot0 + tot1, warp_tot, &cnt);
  const uint32_t gd = block_excl_scan256(dt0 + dt1, warp_tot, &all);
  if (SRC == kVisible && blockIdx.x == 0 && threadIdx.x == 0) *total_out = all;
  lstart[d0] = ls;
  lstart[d1] = ls + tot0;
  gstart[d0] = gd + (d0 <= mask ? hist[(int64_t)d0 * nblocks + blockIdx.x] : 0u);
  gstart[d1] = gd + dt0 + (d1 <= mask ? hist[(int64_t)d1 * nblocks + blockIdx.x] : 0u);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    if ((live >> r) & 1u) {
      const uint32_t dd = (uint32_t)(key[r] >> shift) & mask;
      const uint32_t pos = lstart[dd] + wcnt[w * kRadixBins + dd] + rnk[r];
      sk[pos] = key[r];
      sv[pos] = val[r];
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < (int)cnt; j += kSortThreads) {
    const KT k = sk[j];
    const uint32_t dd = (uint32_t)(k >> shift) & mask;
    const uint32_t g = gstart[dd] + (uint32_t)j - lstart[dd];
    kout[g] = k;
    vout[g] = sv[j];
  }
}

}  // namespace gsb
