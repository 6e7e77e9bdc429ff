// Stable LSD radix sort of (uint32 key, uint32 value) pairs, one pass per
// 8-bit digit, in the onesweep style: one upfront histogram kernel for all
// digit passes, then one kernel per pass that ranks a tile in shared memory,
// resolves the tile's global digit offsets with a decoupled look-back over
// its predecessors, and scatters. Tiles take their index from an atomic
// counter in launch order, so every look-back waits only on tiles that are
// already running; each wait is still bounded and reports kStatusTimeout
// instead of hanging.
//
// Used for the Morton-code sort of the clustering builder
// (src/morton.rs:63-102 sorts the indices by code with a stable sort).
#include "lib_internal.h"

namespace rtbvh {

namespace {

constexpr int kBlock = 256;  // threads per tile == number of digits
// Keys per thread: what a tile costs is the latency of ranking them one after
// another and of the look-back, so few keys take small tiles. LOCB builds: 4
// keys against 15 per thread, 6,400 triangles 464 / 488 us, 20k 529 / 543;
// 8 against 15, 1M triangles 1,453 / 1,482, 4M 3,909 / 3,949. Per pass: 200k
// pairs 15 -> 10 us, 4.2M 53 -> 42.
inline int items_for(size_t n) { return n <= 160000 ? 4 : 8; }
inline size_t tile_for(size_t n) { return (size_t)kBlock * items_for(n); }
// Earlier tiles that a look-back reads at a time.
constexpr int kLook = 4;
constexpr int kWarps = kBlock / 32;
constexpr int kRadix = 256;
// Pairs that one block sorts alone, and its threads. LOCB builds, with tiles
// and alone: 500 triangles 396 / 369 us, 2,000 426 / 399, 4,000 443 /
// 427, 6,400 454 / 452, 8,100 464 / 460.
constexpr int kAloneBlock = 1024;
constexpr size_t kAloneMost = 4 * kAloneBlock;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1u;

struct SortTemp {
  uint32_t* hist;          // passes x 256 (counts, then exclusive offsets)
  uint32_t* tile_counter;  // passes
  uint32_t* lookback;      // passes x tiles x 256
  uint32_t* keys_alt;
  uint32_t* vals_alt;
};

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

inline int passes_for(int bits) { return (bits + 7) / 8; }

SortTemp carve(void* temp, size_t n, int passes) {
  size_t tiles = (n + tile_for(n) - 1) / tile_for(n);
  char* p = static_cast<char*>(temp);
  SortTemp t;
  t.hist = reinterpret_cast<uint32_t*>(p);
  p += align256(4 * kRadix * 4);
  t.tile_counter = reinterpret_cast<uint32_t*>(p);
  p += align256(4 * 4);
  t.lookback = reinterpret_cast<uint32_t*>(p);
  p += align256((size_t)4 * tiles * kRadix * 4);
  t.keys_alt = reinterpret_cast<uint32_t*>(p);
  p += align256(n * 4);
  t.vals_alt = reinterpret_cast<uint32_t*>(p);
  (void)passes;
  return t;
}

__global__ void __launch_bounds__(kBlock)
    k_histogram(const uint32_t* __restrict__ keys, size_t n, int passes, uint32_t* __restrict__ hist) {
  __shared__ uint32_t s_hist[4][kRadix];
  for (int i = threadIdx.x; i < 4 * kRadix; i += kBlock) (&s_hist[0][0])[i] = 0;
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * kBlock + threadIdx.x; i < n; i += (size_t)gridDim.x * kBlock) {
    uint32_t k = __ldg(keys + i);
    for (int p = 0; p < passes; ++p) atomicAdd(&s_hist[p][(k >> (8 * p)) & 0xffu], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p) {
    uint32_t c = s_hist[p][threadIdx.x];
    if (c) atomicAdd(hist + p * kRadix + threadIdx.x, c);
  }
}

// Exclusive scan of each pass's 256 digit counts (one block per pass).
__global__ void __launch_bounds__(kBlock) k_hist_scan(uint32_t* __restrict__ hist) {
  __shared__ uint32_t s_warp[kWarps];
  uint32_t* h = hist + blockIdx.x * kRadix;
  uint32_t v = h[threadIdx.x];
  uint32_t incl = block_inclusive_scan<kBlock>(v, s_warp, nullptr);
  h[threadIdx.x] = incl - v;
}

// Digits are recomputed from the keys and ranks kept in 16 bits: four blocks
// fit an SM (with 15 keys per thread and all of it held it was two).
template <int kItems>
__global__ void __launch_bounds__(kBlock, 4)
    k_onesweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
               uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, size_t n, int shift,
               const uint32_t* __restrict__ digit_offsets, uint32_t* __restrict__ lookback,
               uint32_t* __restrict__ tile_counter, uint32_t* __restrict__ status) {
  constexpr int kTile = kBlock * kItems;
  __shared__ uint32_t s_tile;
  __shared__ int s_fail;
  __shared__ uint32_t s_whist[kWarps][kRadix];
  __shared__ uint32_t s_local_off[kRadix];
  __shared__ uint32_t s_global_base[kRadix];
  __shared__ uint32_t s_warp[kWarps];
  __shared__ uint32_t s_keys[kTile];
  __shared__ uint32_t s_vals[kTile];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_tile = atomicAdd(tile_counter, 1u);
    s_fail = 0;
  }
  for (int i = tid; i < kWarps * kRadix; i += kBlock) (&s_whist[0][0])[i] = 0;
  __syncthreads();
  const size_t tile = s_tile;
  const size_t tile_base = tile * kTile;
  const size_t warp_base = tile_base + (size_t)warp * (kItems * 32);

  uint32_t key[kItems], val[kItems];
  uint16_t rank[kItems];  // below 32 kItems
  const uint32_t in_warp = warp_base >= n ? 0u : (n - warp_base < (size_t)(kItems * 32) ? (uint32_t)(n - warp_base)
                                                                                   : (uint32_t)(kItems * 32));
  auto valid = [&](int k) { return (uint32_t)(k * 32 + lane) < in_warp; };
  auto digit = [&](int k) { return (key[k] >> shift) & 0xffu; };
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    key[k] = valid(k) ? __ldg(keys_in + warp_base + k * 32 + lane) : 0u;
    val[k] = valid(k) ? __ldg(vals_in + warp_base + k * 32 + lane) : 0u;
  }
  const uint32_t lt_mask = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const bool v = valid(k);
    const uint32_t d = v ? digit(k) : (uint32_t)kRadix;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    uint32_t base = 0;
    if (v) base = s_whist[warp][d];
    rank[k] = (uint16_t)(base + __popc(peers & lt_mask));
    __syncwarp();
    if (v && (__ffs(peers) - 1) == lane) s_whist[warp][d] = base + __popc(peers);
    __syncwarp();
  }
  __syncthreads();

  // Thread `tid` owns digit `tid`: warp-exclusive offsets and the tile count.
  const uint32_t d = tid;
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    uint32_t c = s_whist[w][d];
    s_whist[w][d] = run;
    run += c;
  }
  volatile uint32_t* lb = lookback;
  lb[tile * kRadix + d] = (tile == 0 ? kFlagInc : kFlagAgg) | run;
  uint32_t incl = block_inclusive_scan<kBlock>(run, s_warp, nullptr);
  s_local_off[d] = incl - run;

  uint32_t excl = 0;
  if (tile > 0) {
    // kLook earlier tiles per read: with all tiles under way the way back to
    // an inclusive count is as long as the number of tiles in flight
    int64_t j = (int64_t)tile - 1;
    uint32_t spins = 0;
    for (bool done = false; !done;) {
      uint32_t v[kLook];
#pragma unroll
      for (int q = 0; q < kLook; ++q) {
        v[q] = kFlagInc;  // before the first tile
        if (j >= q) v[q] = lb[(size_t)(j - q) * kRadix + d];
      }
      int taken = 0;
#pragma unroll
      for (int q = 0; q < kLook; ++q) {
        if (done || taken != q) continue;
        const uint32_t flag = v[q] & ~kCountMask;
        if (flag == 0u) continue;  // not there yet: read again from this tile
        excl += v[q] & kCountMask;
        ++taken;
        done = flag == kFlagInc;
      }
      j -= taken;
      if (!done && taken == 0) {
        if (++spins > kSpinLimit) {
          atomicOr(status, kStatusTimeout);
          s_fail = 1;
          break;
        }
        __nanosleep(32);
      }
    }
    lb[tile * kRadix + d] = kFlagInc | (excl + run);
  }
  s_global_base[d] = __ldg(digit_offsets + d) + excl;
  __syncthreads();
  if (s_fail) return;

#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (valid(k)) {
      const uint32_t dk = digit(k), pos = s_local_off[dk] + s_whist[warp][dk] + rank[k];
      s_keys[pos] = key[k];
      s_vals[pos] = val[k];
    }
  }
  __syncthreads();
  const size_t remaining = n - tile_base;
  const uint32_t tile_count = remaining < (size_t)kTile ? (uint32_t)remaining : (uint32_t)kTile;
  for (uint32_t i = tid; i < tile_count; i += kBlock) {
    uint32_t k = s_keys[i];
    uint32_t dd = (k >> shift) & 0xffu;
    size_t g = (size_t)s_global_base[dd] + (i - s_local_off[dd]);
    if (g < n) {
      keys_out[g] = k;
      vals_out[g] = s_vals[i];
    } else {
      atomicOr(status, kStatusBadIndex);
    }
  }
}

// All passes over at most kAloneBlock * kItems pairs in one block: the pairs
// stay in registers (k-th row of a warp's run, lane) and change places through
// shared memory, which holds the warps' digit counts before that. What bounds
// it is the issue of the ranking, 32 warps on one SM. Instead of six launches
// and three memsets.
template <int kItems>
__global__ void __launch_bounds__(kAloneBlock)
    k_sort_alone(uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n, int passes) {
  constexpr int kRun = kItems * 32, kRows = kAloneBlock / 32;
  __shared__ uint32_t s_buf[kAloneBlock * kItems > kRows * kRadix / 2 ? kAloneBlock * kItems : kRows * kRadix / 2];
  __shared__ uint32_t s_off[kRadix];
  __shared__ uint32_t s_warp[kAloneBlock / 32];
  uint16_t* const whist = reinterpret_cast<uint16_t*>(s_buf);  // [warp][digit], counts and offsets up to n
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t first = warp * kRun + lane, lt_mask = (1u << lane) - 1u;
  uint32_t key[kItems], val[kItems];
  uint16_t pos[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const uint32_t i = first + k * 32;
    key[k] = i < n ? keys[i] : 0u;
    val[k] = i < n ? vals[i] : 0u;
  }
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    for (uint32_t i = tid; i < kRows * kRadix / 2; i += kAloneBlock) s_buf[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const bool v = first + k * 32 < n;
      const uint32_t d = (key[k] >> shift) & 0xffu;
      uint32_t peers = __ballot_sync(0xffffffffu, v);
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
      }
      uint32_t base = 0;
      if (v) base = whist[warp * kRadix + d];
      pos[k] = (uint16_t)(base + __popc(peers & lt_mask));
      __syncwarp();
      if (v && (peers & lt_mask) == 0u) whist[warp * kRadix + d] = (uint16_t)(base + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t run = 0;
    if (tid < (uint32_t)kRadix) {
#pragma unroll 8
      for (int w = 0; w < kRows; ++w) {
        const uint32_t c = whist[w * kRadix + tid];
        whist[w * kRadix + tid] = (uint16_t)run;
        run += c;
      }
    }
    const uint32_t incl = block_inclusive_scan<kAloneBlock>(run, s_warp, nullptr);
    if (tid < (uint32_t)kRadix) s_off[tid] = incl - run;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t d = (key[k] >> shift) & 0xffu;
      pos[k] = (uint16_t)(pos[k] + s_off[d] + whist[warp * kRadix + d]);
    }
    if (p + 1 == passes) break;
    __syncthreads();
    auto exchange = [&](uint32_t (&x)[kItems]) {
#pragma unroll
      for (int k = 0; k < kItems; ++k)
        if (first + k * 32 < n) s_buf[pos[k]] = x[k];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kItems; ++k) x[k] = first + k * 32 < n ? s_buf[first + k * 32] : 0u;
      __syncthreads();
    };
    exchange(key);
    exchange(val);
  }
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (first + k * 32 < n) {
      keys[pos[k]] = key[k];
      vals[pos[k]] = val[k];
    }
  }
}

}  // namespace

size_t radix_sort_temp_bytes(size_t n) {
  size_t tiles = (n + tile_for(n) - 1) / tile_for(n);
  return align256(4 * kRadix * 4) + align256(16) + align256((size_t)4 * tiles * kRadix * 4) + 2 * align256(n * 4) +
         256;
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, size_t n, int bits, void* temp, size_t temp_bytes,
                             uint32_t* status, cudaStream_t s) {
  if (n <= 1) return cudaSuccess;
  if (n > kCountMask || temp_bytes < radix_sort_temp_bytes(n)) return cudaErrorInvalidValue;
  const int passes = passes_for(bits);
  if (passes == 0) return cudaSuccess;
  if (n <= kAloneMost) {
    auto alone = n <= 2 * kAloneBlock ? k_sort_alone<2> : k_sort_alone<4>;
    alone<<<1, kAloneBlock, 0, s>>>(keys, vals, (uint32_t)n, passes);
    return cudaGetLastError();
  }
  const size_t tiles = (n + tile_for(n) - 1) / tile_for(n);
  SortTemp t = carve(temp, n, passes);
  cudaError_t e;
  if ((e = cudaMemsetAsync(t.hist, 0, 4 * kRadix * 4, s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(t.tile_counter, 0, 16, s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(t.lookback, 0, (size_t)passes * tiles * kRadix * 4, s)) != cudaSuccess) return e;
  unsigned hblocks = (unsigned)((n + kBlock - 1) / kBlock);
  unsigned cap = (unsigned)sm_count() * 4u;
  if (hblocks > cap) hblocks = cap;
  k_histogram<<<hblocks, kBlock, 0, s>>>(keys, n, passes, t.hist);
  k_hist_scan<<<passes, kBlock, 0, s>>>(t.hist);
  auto sweep = items_for(n) == 4 ? k_onesweep<4> : k_onesweep<8>;
  uint32_t *kin = keys, *vin = vals, *kout = t.keys_alt, *vout = t.vals_alt;
  for (int p = 0; p < passes; ++p) {
    sweep<<<(unsigned)tiles, kBlock, 0, s>>>(kin, vin, kout, vout, n, 8 * p, t.hist + p * kRadix,
                                                  t.lookback + (size_t)p * tiles * kRadix, t.tile_counter + p,
                                                  status);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  if (kin != keys) {
    if ((e = cudaMemcpyAsync(keys, kin, n * 4, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(vals, vin, n * 4, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

}  // namespace rtbvh
