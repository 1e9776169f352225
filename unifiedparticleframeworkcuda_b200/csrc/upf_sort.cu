// upf_sort.cu — stable LSD radix sort of (key, value) pairs, Morton keys and
// cell ranges.
//
// Replaces the reference's 2006 SDK sort (RadixSum / RadixPrefixSum /
// RadixAddOffsetsAndShuffle, src/gpu/radixsort_kernel.cu:64-540, driver
// src/gpu/particles.cu:31-60), which runs a fixed 48-CTA grid. Here each pass
// is three launches sized to the input, one CTA per tile of 512, 2048 or 8192
// keys (radix_tile_keys: the smallest tile that needs at most kRadixTileCap
// tiles):
//   upsweep   per-tile digit histograms (shared-memory atomics)
//   scan      per digit, exclusive scan of its row of tile counts (one CTA
//             per digit) and the digit's total
//   downsweep per-tile stable ranking with warp votes (each warp owns
//             a contiguous segment of 32, 128 or 512 keys, rounds run in key
//             order), a local sort through shared memory, and coalesced runs
//             to global memory.
// Stability: warps own consecutive segments and rank in order, so equal
// digits keep their input order; an LSD sort of stable passes is stable.
// Ranks come from a vote per bit of the digit, not from match.any, whose cost
// grows with the distinct values in a warp (four passes of 262,144 pairs 38.8
// against 43.0 us, 1,048,576 62.5 / 83.4, 5,204,419 264 / 360).
// Up to 32,768 keys one CTA or one cluster runs all passes in one launch
// (k_radix_cluster), without the gaps between 12 launches; above, the ranking
// of more pairs an SM costs more than the gaps.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <mutex>

#include "upf_common.cuh"
#include "upf_internal.h"

namespace upf {

namespace {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kThreads = 512;               // 16 warps
constexpr int kWarps = kThreads / 32;
static_assert(kRadix == (int)kRadixDigits, "scratch layout constants");

// The lanes of the warp (all of it active) whose digit is d: a vote per bit.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d) {
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < kRadixBits; ++b) {
    const bool set = (d >> b) & 1u;
    const uint32_t with = __ballot_sync(0xffffffffu, set);
    peers &= set ? with : ~with;
  }
  return peers;
}

// kItems keys per lane: a warp ranks 32 * kItems consecutive keys, a tile is
// kWarps warps' segments
template <int kItems>
__global__ void __launch_bounds__(kThreads) k_upsweep(const uint32_t* __restrict__ keys, uint32_t n,
                                                       int shift, uint32_t ntiles,
                                                       uint32_t* __restrict__ counts) {
  constexpr int kTile = kWarps * 32 * kItems;
  __shared__ uint32_t hist[kRadix];
  for (int d = threadIdx.x; d < kRadix; d += kThreads) hist[d] = 0;
  __syncthreads();
  const uint32_t base = blockIdx.x * (uint32_t)kTile;
#pragma unroll 4
  for (int r = 0; r < kTile / kThreads; ++r) {
    uint32_t i = base + r * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&hist[(keys[i] >> shift) & (kRadix - 1)], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < kRadix; d += kThreads) counts[(size_t)d * ntiles + blockIdx.x] = hist[d];
}

// Exclusive scan of each digit's row of tile counts, one CTA of 256 threads
// per digit: counts[d][t] becomes the number of keys with digit d in tiles
// before t, and totals[d] the digit's count over all tiles. The downsweep
// adds the digit's base (the exclusive scan of the totals).
__global__ void __launch_bounds__(256) k_scan_rows(uint32_t* __restrict__ counts, uint32_t ntiles,
                                                   uint32_t* __restrict__ totals) {
  __shared__ uint32_t warp_sums[8];
  __shared__ uint32_t carry;
  uint32_t* row = counts + (size_t)blockIdx.x * ntiles;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t base = 0; base < ntiles; base += 256 * 4) {
    uint32_t v[4];
    const uint32_t idx0 = base + threadIdx.x * 4;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = (idx0 + k < ntiles) ? row[idx0 + k] : 0u;
      s += v[k];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const uint32_t w = lane < 8 ? warp_sums[lane] : 0u;
      uint32_t wi = w;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      if (lane < 8) warp_sums[lane] = wi - w;  // exclusive
    }
    __syncthreads();
    uint32_t run = carry + warp_sums[warp] + (incl - s);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (idx0 + k < ntiles) row[idx0 + k] = run;
      run += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 255) carry = run;
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template <int kItems>
constexpr size_t down_smem() {
  return sizeof(uint32_t) * (kWarps * kRadix + 2 * (kWarps * 32 * kItems) + 3 * kRadix);
}

template <bool kIotaValues, int kItems>
__global__ void __launch_bounds__(kThreads) k_downsweep(const uint32_t* __restrict__ keys_in,
                                                         const uint32_t* __restrict__ vals_in,
                                                         uint32_t* __restrict__ keys_out,
                                                         uint32_t* __restrict__ vals_out, uint32_t n,
                                                         int shift, uint32_t ntiles,
                                                         const uint32_t* __restrict__ counts,
                                                         const uint32_t* __restrict__ totals) {
  constexpr int kItemsPerLane = kItems;
  constexpr int kWarpItems = 32 * kItems;
  constexpr int kTile = kWarps * kWarpItems;
  extern __shared__ uint32_t smem[];
  uint32_t* whist = smem;                                  // [kWarps][kRadix]
  uint32_t* skeys = whist + kWarps * kRadix;               // [kItems * 512]
  uint32_t* svals = skeys + kTile;                         // [kTile]
  uint32_t* digit_off = svals + kTile;                     // [kRadix] tile-local digit offsets
  uint32_t* gbase = digit_off + kRadix;                    // [kRadix] global bases
  uint32_t* dbase = gbase + kRadix;                        // [kRadix] digit bases over all tiles

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = threadIdx.x; d < kWarps * kRadix; d += kThreads) whist[d] = 0;
  __syncthreads();

  const uint32_t tile_base = blockIdx.x * (uint32_t)kTile;
  const uint32_t seg_base = tile_base + warp * kWarpItems;
  uint32_t* wh = whist + warp * kRadix;
  uint32_t k[kItemsPerLane], v[kItemsPerLane];
  uint32_t local[kItemsPerLane];
  const uint32_t lt = lanemask_lt();
#pragma unroll
  for (int r = 0; r < kItemsPerLane; ++r) {
    uint32_t i = seg_base + r * 32 + lane;
    bool valid = i < n;
    k[r] = valid ? keys_in[i] : 0xffffffffu;
    v[r] = valid ? (kIotaValues ? i : vals_in[i]) : 0u;
    uint32_t d = (k[r] >> shift) & (kRadix - 1);
    const uint32_t peers = digit_peers(d) & __ballot_sync(0xffffffffu, valid);
    const uint32_t rank = __popc(peers & lt), prior = wh[d];
    local[r] = prior + rank;
    __syncwarp();
    if (valid && rank == 0) wh[d] = prior + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: exclusive prefix over warps, and the tile's digit totals
  for (int d = threadIdx.x; d < kRadix; d += kThreads) {
    uint32_t acc = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      uint32_t t = whist[w * kRadix + d];
      whist[w * kRadix + d] = acc;
      acc += t;
    }
    digit_off[d] = acc;  // total for now
    gbase[d] = counts[(size_t)d * ntiles + blockIdx.x];
    dbase[d] = totals[d];
  }
  __syncthreads();
  // digit bases: exclusive scan of the 256 digit totals (warp 1, 8 per lane)
  if (warp == 1) {
    uint32_t t[8], s = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      t[q] = dbase[lane * 8 + q];
      s += t[q];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    uint32_t run = incl - s;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      gbase[lane * 8 + q] += run;
      run += t[q];
    }
  }
  // the tile's digit offsets: exclusive scan of its 256 digit totals (warp 0)
  if (warp == 0) {
    uint32_t t[8], s = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      t[q] = digit_off[lane * 8 + q];
      s += t[q];
    }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    uint32_t run = incl - s;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      digit_off[lane * 8 + q] = run;
      run += t[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kItemsPerLane; ++r) {
    uint32_t i = seg_base + r * 32 + lane;
    if (i < n) {
      uint32_t d = (k[r] >> shift) & (kRadix - 1);
      uint32_t pos = digit_off[d] + whist[warp * kRadix + d] + local[r];
      skeys[pos] = k[r];
      svals[pos] = v[r];
    }
  }
  __syncthreads();
  const uint32_t tile_n = (n - tile_base < (uint32_t)kTile) ? (n - tile_base) : (uint32_t)kTile;
  for (uint32_t i = threadIdx.x; i < tile_n; i += kThreads) {
    uint32_t key = skeys[i];
    uint32_t d = (key >> shift) & (kRadix - 1);
    uint32_t g = gbase[d] + (i - digit_off[d]);
    keys_out[g] = key;
    vals_out[g] = svals[i];
  }
}

constexpr int kSmallThreads = 512;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallGroups = kSmallThreads / kRadix;  // of eight warps
constexpr int kSegmentCtas = 8, kSegmentItems = 16;
static_assert(kSegmentCtas * kSegmentItems * kSmallThreads == kRadixSegmentMax, "segments");

template <int kItems>
constexpr size_t cluster_smem() {
  return sizeof(uint2) * kSmallThreads * kItems +
         sizeof(uint32_t) * (kSmallWarps * kRadix + kRadix + 2 * kSmallGroups * kRadix);
}

// All passes of a sort by one cluster of kCtas CTAs (one CTA: no cluster), each
// of which holds rounds * 512 (at most kItems * 512) consecutive pairs of the
// current order in registers: round r of a thread is the pair at lane + 32 (r +
// rounds * warp). A pass ranks them as k_downsweep does, adds the digit counts
// of all CTAs (read from their shared memory) to the places of its own, and
// sends every pair to the shared memory of the CTA that holds its place.
// `load(i, k, v)` fetches pair i, `store(i, k, v)` takes the i-th of the order.
template <int kCtas, int kItems, class Load, class Store>
__device__ __forceinline__ void sort_in_cluster(uint32_t rounds, int passes, Load&& load, Store&& store) {
  const uint32_t tile = kSmallThreads * rounds;
  // x / rounds of x < 256, as the product with the rounded-up 16-bit inverse
  const uint32_t inverse = (65536u + rounds - 1) / rounds;
  static_assert(kCtas * kItems <= 256 && kItems <= 16, "inverse");
  extern __shared__ uint2 pair_mem[];
  uint2* const pairs = pair_mem;                                       // [kTile]
  uint32_t* const whist = reinterpret_cast<uint32_t*>(pairs + kSmallThreads * kItems);  // [kSmallWarps][kRadix]
  uint32_t* const count = whist + kSmallWarps * kRadix;                // [kRadix] this CTA's digit counts
  uint32_t* const part = count + kRadix;                               // [kSmallGroups][kRadix] the groups' counts
  uint32_t* const base = part + kSmallGroups * kRadix;                 // [kSmallGroups][kRadix] a group's first place
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const auto barrier = [&] {
    if constexpr (kCtas > 1)
      cluster.sync();
    else
      __syncthreads();
  };
  const uint32_t cta = kCtas > 1 ? cluster.block_rank() : 0u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = lanemask_lt();
  const uint32_t seg = warp * 32 * rounds + lane;
  uint32_t k[kItems], v[kItems];
  uint32_t local[(kItems + 1) / 2];  // 16 bits each
#pragma unroll
  for (int r = 0; r < kItems; ++r)
    if ((uint32_t)r < rounds) load(cta * tile + seg + r * 32, k[r], v[r]);
  uint32_t* const wh = whist + warp * kRadix;
  for (int shift = 0; shift < passes * kRadixBits; shift += kRadixBits) {
#pragma unroll
    for (int d = lane; d < kRadix; d += 32) wh[d] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if ((uint32_t)r >= rounds) break;
      const uint32_t d = (k[r] >> shift) & (kRadix - 1);
      const uint32_t peers = digit_peers(d);
      const uint32_t rank = __popc(peers & lt), prior = wh[d];
      local[r / 2] = r & 1 ? local[r / 2] | (prior + rank) << 16 : prior + rank;
      __syncwarp();
      if (rank == 0) wh[d] = prior + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over the warps of each group of eight, the
    // groups' counts and their sum
    {
      const int d = threadIdx.x & (kRadix - 1), g = threadIdx.x / kRadix;
      uint32_t run = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const uint32_t t = whist[(g * 8 + w) * kRadix + d];
        whist[(g * 8 + w) * kRadix + d] = run;
        run += t;
      }
      part[g * kRadix + d] = run;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
      uint32_t run = 0;
#pragma unroll
      for (int g = 0; g < kSmallGroups; ++g) run += part[g * kRadix + threadIdx.x];
      count[threadIdx.x] = run;
    }
    barrier();
    // the CTAs' counts: all of a digit's keys, and those of the CTAs before
    if (threadIdx.x < kRadix) {
      uint32_t all = 0, before = 0;
#pragma unroll
      for (int c = 0; c < kCtas; ++c) {
        const uint32_t t = kCtas > 1 ? cluster.map_shared_rank(count, c)[threadIdx.x] : count[threadIdx.x];
        all += t;
        if (c < (int)cta) before += t;
      }
      // exclusive scan of the 256 totals: in the warp, then over eight warps
      uint32_t incl = all;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      __shared__ uint32_t warp_total[kRadix / 32];
      if (lane == 31) warp_total[warp] = incl;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      uint32_t run = incl - all + before;
#pragma unroll
      for (int w = 0; w < kRadix / 32; ++w)
        if (w < warp) run += warp_total[w];
#pragma unroll
      for (int g = 0; g < kSmallGroups; ++g) {
        base[g * kRadix + threadIdx.x] = run;
        run += part[g * kRadix + threadIdx.x];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if ((uint32_t)r >= rounds) break;
      const uint32_t d = (k[r] >> shift) & (kRadix - 1);
      const uint32_t at = base[(warp / 8) * kRadix + d] + wh[d] + (local[r / 2] >> 16 * (r & 1) & 0xffffu);
      const uint32_t owner = kCtas > 1 ? (at / kSmallThreads * inverse) >> 16 : 0u;
      uint2* const to = kCtas > 1 ? cluster.map_shared_rank(pairs, owner) : pairs;
      to[at - owner * tile] = make_uint2(k[r], v[r]);
    }
    barrier();
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
      if ((uint32_t)r >= rounds) break;
      const uint2 p = pairs[seg + r * 32];
      k[r] = p.x;
      v[r] = p.y;
    }
  }
#pragma unroll
  for (int r = 0; r < kItems; ++r)
    if ((uint32_t)r < rounds) store(cta * tile + seg + r * 32, k[r], v[r]);
}

// Up to kCtas * kItems * 512 pairs.
// Bound by the ranking (0.6 us a round of 16 warps, some 70 instructions a
// warp) and the barriers (0.3 us each across a cluster). Four passes, us, in
// one launch and in twelve: 900 pairs 5.5 and 25, 1,728 8.3, 4,096 11.3, 8,192
// 11.8, 16,384 16.6 and 25.2, 32,768 on 16 CTAs 21.4 and 25.9; on 8 CTAs 26.0,
// and 50,000 on 16 31.6 and 26.3. CTAs of 1,024 threads are 1 to 2 us longer
// (more rows of counts to add up), pairs put in order in the CTA before they
// are sent not shorter.
template <bool kIotaValues, int kCtas, int kItems>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kSmallThreads)
    k_radix_cluster(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n, int passes) {
  sort_in_cluster<kCtas, kItems>(
      kItems, passes,
      [&](uint32_t i, uint32_t& k, uint32_t& v) {
        k = i < n ? keys[i] : 0xffffffffu;  // beyond the last key: behind all others in every pass
        v = i < n ? (kIotaValues ? i : vals[i]) : 0u;
      },
      [&](uint32_t i, uint32_t k, uint32_t v) {
        if (i < n) {
          keys[i] = k;
          vals[i] = v;
        }
      });
}

// Segments of one array, each sorted by a cluster of its own: perm gets the
// index (in the whole array) of each place's key; the keys stay as they are.
// Against one sort of the whole array and a further pass by segment (24 MB of
// keys and indices in and out five times): a batch of 256 scenes, 5.2 million
// slots, sorted and reordered in 0.41 ms, 0.57 before; 12 scenes of 2,048 to
// 16,384 0.039 and 0.098 (fifteen launches). One scene of 65,536 alone takes
// 45 us either way; a longer one does not fit the cluster's registers.
template <int kItems>
__global__ void __cluster_dims__(kSegmentCtas, 1, 1) __launch_bounds__(kSmallThreads, 2)
    k_radix_segments(const uint2* __restrict__ segments, const uint32_t* __restrict__ keys,
                     uint32_t* __restrict__ perm) {
  const uint2 seg = segments[blockIdx.x / kSegmentCtas];  // first, count
  constexpr uint32_t round = kSegmentCtas * kSmallThreads;
  sort_in_cluster<kSegmentCtas, kItems>(
      (seg.y + round - 1) / round, 32 / kRadixBits,
      [&](uint32_t i, uint32_t& k, uint32_t& v) {
        k = i < seg.y ? keys[seg.x + i] : 0xffffffffu;
        v = seg.x + i;
      },
      [&](uint32_t i, uint32_t, uint32_t v) {
        if (i < seg.y) perm[seg.x + i] = v;
      });
}

// The one-launch forms: the largest count of each, in order.
struct SmallForm {
  uint32_t max;
  const void* iota;
  const void* given;
  uint32_t ctas;
  size_t smem;
};
template <int kCtas, int kItems>
constexpr SmallForm small_form() {
  return {(uint32_t)kCtas * kSmallThreads * kItems, (const void*)k_radix_cluster<true, kCtas, kItems>,
          (const void*)k_radix_cluster<false, kCtas, kItems>, (uint32_t)kCtas, cluster_smem<kItems>()};
}
const SmallForm kSmallForms[] = {
    small_form<1, 2>(), small_form<1, 4>(), small_form<8, 2>(), small_form<8, 4>(), small_form<16, 4>(),};

// The largest count the one-launch forms take on the current device: a
// cluster of 16 needs as many free SMs in one group of the chip, which a
// partition of it need not have. Set by radix_init.
constexpr int kMaxDevices = 64;
uint32_t g_small_max[kMaxDevices] = {};
uint32_t small_max() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  return __atomic_load_n(&g_small_max[dev], __ATOMIC_ACQUIRE);
}

cudaError_t small_init(int dev) {
  const cudaError_t e = cudaFuncSetAttribute(k_radix_segments<kSegmentItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)cluster_smem<kSegmentItems>());
  if (e != cudaSuccess) return e;
  uint32_t fits = 0;
  for (const SmallForm& f : kSmallForms) {
    int clusters = 0;
    for (const void* k : {f.iota, f.given}) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem);
      if (e == cudaSuccess && f.ctas > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.ctas);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = f.smem;
    cudaLaunchAttribute size = {};
    size.id = cudaLaunchAttributeClusterDimension;
    size.val.clusterDim.x = f.ctas;
    size.val.clusterDim.y = size.val.clusterDim.z = 1;
    cfg.attrs = &size;
    cfg.numAttrs = 1;
    if (f.ctas > 1 && (cudaOccupancyMaxActiveClusters(&clusters, f.given, &cfg) != cudaSuccess || clusters < 1)) {
      cudaGetLastError();
      break;
    }
    fits = f.max;
  }
  if (dev >= 0 && dev < kMaxDevices) __atomic_store_n(&g_small_max[dev], fits, __ATOMIC_RELEASE);
  return cudaSuccess;
}

}  // namespace

// scratch layout: keys_alt[pad64(n)] | vals_alt[pad64(n)] | counts[256 * tiles]
size_t radix_temp_words(uint32_t n) {
  size_t pad = ((size_t)n + 63) & ~size_t(63);
  return 2 * pad + radix_count_words(n);
}

size_t radix_temp_bytes(uint32_t n) { return radix_temp_words(n) * sizeof(uint32_t); }

// Opt the kernels of over 48 KB into their dynamic shared memory on the
// current device, once per device (before any launch on it, and so before
// any stream capture that launches it).
cudaError_t radix_init() {
  static std::mutex mu;
  static bool done[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (dev >= 0 && dev < kMaxDevices && done[dev]) return cudaSuccess;
  e = cudaFuncSetAttribute(k_downsweep<true, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)down_smem<16>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_downsweep<false, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)down_smem<16>());
  if (e == cudaSuccess) e = small_init(dev);
  if (e == cudaSuccess && dev >= 0 && dev < kMaxDevices) done[dev] = true;
  return e;
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt,
                             uint32_t* counts, uint32_t n, int key_bits, bool iota_values,
                             cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t ntiles = radix_tiles(n);
  const uint32_t tile = radix_tile_keys(n);
  // the digit totals follow the [256][ntiles] counts
  uint32_t* totals = counts + (size_t)kRadix * ntiles;
  int passes = (key_bits + kRadixBits - 1) / kRadixBits;
  if (passes < 1) passes = 1;
  if (n <= small_max()) {
    const SmallForm* f = kSmallForms;
    while (n > f->max) ++f;
    void* args[] = {&keys, &vals, &n, &passes};
    return cudaLaunchKernel(iota_values ? f->iota : f->given, dim3(f->ctas), dim3(kSmallThreads), args, f->smem, st);
  }
  uint32_t *ki = keys, *vi = vals, *ko = keys_alt, *vo = vals_alt;
  for (int p = 0; p < passes; ++p) {
    int shift = p * kRadixBits;
    const bool iota = p == 0 && iota_values;
#define UPF_PASS(I)                                                                                          \
  k_upsweep<I><<<ntiles, kThreads, 0, st>>>(ki, n, shift, ntiles, counts);                                   \
  k_scan_rows<<<kRadix, 256, 0, st>>>(counts, ntiles, totals);                                               \
  if (iota)                                                                                                  \
    k_downsweep<true, I><<<ntiles, kThreads, down_smem<I>(), st>>>(ki, vi, ko, vo, n, shift, ntiles, counts,  \
                                                                    totals);                                  \
  else                                                                                                       \
    k_downsweep<false, I><<<ntiles, kThreads, down_smem<I>(), st>>>(ki, vi, ko, vo, n, shift, ntiles, counts, \
                                                                     totals);
    if (tile == 8192u) {
      UPF_PASS(16)
    } else if (tile == 2048u) {
      UPF_PASS(4)
    } else {
      UPF_PASS(1)
    }
#undef UPF_PASS
    uint32_t* t;
    t = ki; ki = ko; ko = t;
    t = vi; vi = vo; vo = t;
  }
  // an odd number of passes leaves the result in the alternate buffers
  if (passes & 1) {
    cudaError_t e = cudaMemcpyAsync(keys, ki, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(vals, vi, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t radix_sort_segments(const uint2* segments, uint32_t count, const uint32_t* keys, uint32_t* perm,
                                cudaStream_t st) {
  if (!count) return cudaSuccess;
  k_radix_segments<kSegmentItems><<<count * kSegmentCtas, kSmallThreads, cluster_smem<kSegmentItems>(), st>>>(
      segments, keys, perm);
  return cudaGetLastError();
}

bool radix_segments_fit(uint32_t longest) { return longest <= kRadixSegmentMax && small_max() >= 16384u; }

int radix_launches(uint32_t n, int key_bits) {
  if (n <= small_max()) return 1;
  int passes = (key_bits + kRadixBits - 1) / kRadixBits;
  if (passes < 1) passes = 1;
  return 3 * passes;
}

// ---- Morton keys ------------------------------------------------------------
__global__ void k_morton_keys(const float4* __restrict__ pos, uint32_t n, float3 origin, float3 scales,
                              uint32_t* __restrict__ keys) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) keys[i] = morton_key(pos[i], origin, scales);
}

cudaError_t morton_keys(const float4* pos, uint32_t n, float3 origin, float3 scales, uint32_t* keys,
                        cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_morton_keys<<<(n + 255) / 256, 256, 0, st>>>(pos, n, origin, scales, keys);
  return cudaGetLastError();
}

// ---- cell ranges ------------------------------------------------------------
// ClearIndexArrays + CalculateBlocksKernel (src/gpu/particles_kernel.cu:656-726)
// become a boundary scan over the sorted keys: deterministic, no atomics.
__global__ void k_cell_ranges(const uint32_t* __restrict__ keys, uint32_t n, int shift, uint32_t ncells,
                              uint32_t* __restrict__ start, uint32_t* __restrict__ end) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t c = keys[i] >> shift;
  if (c >= ncells) return;
  if (i == 0 || (keys[i - 1] >> shift) != c) start[c] = i;
  if (i == n - 1 || (keys[i + 1] >> shift) != c) end[c] = i + 1;
}

cudaError_t cell_ranges(const uint32_t* keys, uint32_t n, int shift, uint32_t ncells, uint32_t* start,
                        uint32_t* end, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(start, 0, sizeof(uint32_t) * ncells, st);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(end, 0, sizeof(uint32_t) * ncells, st);
  if (e != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  k_cell_ranges<<<(n + 255) / 256, 256, 0, st>>>(keys, n, shift, ncells, start, end);
  return cudaGetLastError();
}

}  // namespace upf
