// Locally-ordered clustering build (src/builders/locb.rs) on the GPU.
//
// Pipeline: primitive boxes -> world box (Aabb::union_of_list) -> 30-bit
// Morton codes of the centres -> stable radix sort -> leaves (sorted boxes
// + 1e-4) -> clustering levels until one node is left.
//
// A level of m nodes [begin, end) has two phases with a barrier after each:
//   A. for a contiguous chunk per block: the nearest neighbour of every
//      node inside the window [max(begin, i-14), min(end, i+15)) by the
//      half area of the union, first (lowest index) minimum wins -- boxes
//      staged in shared memory, the neighbours of a 14-node halo on either
//      side recomputed -- so the block knows its nodes' merge flags
//      (i < j, nb[j] == i) and counts them at once;
//   B. the prefix of the blocks' counts and the scatter of parents,
//      unmerged nodes (next level) and children (final node array).
// Levels of more than kClusterCap nodes per block of a cluster run in ONE
// cooperative launch with grid barriers and the levels in global memory
// (k_locb_levels); from there on one thread-block cluster keeps the whole
// level in its blocks' shared memory (cluster_levels): halos are read from and
// parents written to the neighbours' shared memory, and the barriers are the
// cluster's. Levels of at most 256 nodes (kClusterAlone) are one block's, of at
// most 32 one warp's (warp_levels).
// Many meshes: the same two forms with a cluster per mesh (k_locb_forest).
// Node positions follow the reference exactly (locb.rs:178-215), so the
// output is bit-identical to the reference's node array.
#include <algorithm>
#include <cstdio>

#include "lib_internal.h"
#include "per_device.h"

namespace rtbvh {

namespace {

constexpr int kBlock = 256;
constexpr int kRadius = 14;       // LocallyOrderedClusteringBuilder::search_radius
struct LocbParams {
  DAabb* lvl[2];
  DAabb* final_nodes;
  uint32_t* nb;
  uint32_t* blocksum;
  GridBarrier* bar;
  uint32_t* status;
  uint32_t* info;  // levels run, then begin, end and level buffer of the first cluster level
  uint32_t n;
  uint32_t stop;   // k_locb_levels runs the levels of more nodes than this
};

struct SBox {
  float mn[3], mx[3];
};

// half_area(union(a, b)); only the comparison of these values matters, so
// native min/max are fine here (a -0/+0 difference cannot change an order).
__device__ __forceinline__ float union_half_area(const SBox& a, const SBox& b) {
  return half_area(fminf(a.mn[0], b.mn[0]), fminf(a.mn[1], b.mn[1]), fminf(a.mn[2], b.mn[2]),
                   fmaxf(a.mx[0], b.mx[0]), fmaxf(a.mx[1], b.mx[1]), fmaxf(a.mx[2], b.mx[2]));
}

// Merge state of node i, kept in the top bits of its nb word in the levels in
// global memory (neighbour indices are below 2^30): kPairHead when i < nb[i]
// and nb[nb[i]] == i (i heads a merged pair: the merge flag of
// locb.rs:159-167), kPairTail when nb[i] < i and nb[nb[i]] == i.
constexpr uint32_t kPairHead = 1u << 30;
constexpr uint32_t kPairTail = 2u << 30;
constexpr uint32_t kNbMask = (1u << 30) - 1u;
constexpr int kHalo = 2 * kRadius;  // boxes a tile stages on each side

// A window of boxes in shared memory: {min, count} and {max, left_first} of
// window index i at (i >> 1) + (i & 1) * half, so that threads that take two
// neighbouring nodes each read consecutive float4s. What bounds the search is
// shared-memory bandwidth: 28 boxes of 32 bytes per node when every thread
// takes one, 30 per two nodes here. 1M triangles: the 16 levels above
// 32,768 nodes take 443 us (before: 29 levels down to 2,048 nodes 655 us).
struct BoxWindow {
  float4 *a, *b;
  int half;
  __device__ __forceinline__ int at(int i) const { return (i >> 1) + (i & 1) * half; }
  __device__ __forceinline__ SBox box(int i) const {
    const float4 u = a[at(i)], v = b[at(i)];
    SBox r;
    r.mn[0] = u.x; r.mn[1] = u.y; r.mn[2] = u.z;
    r.mx[0] = v.x; r.mx[1] = v.y; r.mx[2] = v.z;
    return r;
  }
  __device__ __forceinline__ DAabb node(int i) const {
    const float4 u = a[at(i)], v = b[at(i)];
    DAabb r;
    r.min[0] = u.x; r.min[1] = u.y; r.min[2] = u.z; r.count = __float_as_int(u.w);
    r.max[0] = v.x; r.max[1] = v.y; r.max[2] = v.z; r.left_first = __float_as_int(v.w);
    return r;
  }
  __device__ __forceinline__ void set(int i, float4 u, float4 v) const {
    a[at(i)] = u;
    b[at(i)] = v;
  }
  // outside the level: the infinite box, whose unions have infinite area and
  // never win
  __device__ __forceinline__ void set_outside(int i) const {
    const float inf = __int_as_float(0x7f800000);
    set(i, make_float4(-inf, -inf, -inf, 0.0f), make_float4(inf, inf, inf, 0.0f));
  }
};

// Nearest neighbours of the window nodes i0 (even, >= 14) and i0 + 1: the
// first minimum over the 14 nodes on either side, as window indices (-1: no
// distance below f32::MAX). L neighbouring lanes share a pair; every lane of
// the group gets the result.
template <int L>
__device__ __forceinline__ void nearest_pair(const BoxWindow& w, int i0, int (&bj)[2]) {
  const SBox x0 = w.box(i0), x1 = w.box(i0 + 1);
  const int l = threadIdx.x & (L - 1);
  float b0 = 3.40282347e+38f, b1 = 3.40282347e+38f;
  int j0 = -1, j1 = -1;
  constexpr int N = 2 * kRadius + 2;  // candidates i0 - 14 .. i0 + 15
  auto test = [&](int k) {
    const int c = i0 - kRadius + k;
    const SBox y = w.box(c);
    const float d0 = union_half_area(x0, y), d1 = union_half_area(x1, y);
    if (k != kRadius && k != N - 1 && d0 < b0) {
      b0 = d0;
      j0 = c;
    }
    if (k != 0 && k != kRadius + 1 && d1 < b1) {
      b1 = d1;
      j1 = c;
    }
  };
  if (L == 1) {
#pragma unroll 10
    for (int k = 0; k < N; ++k) test(k);
  } else {
    // the lanes past the last candidate repeat it (an equal distance never
    // replaces an equal one)
#pragma unroll
    for (int k0 = 0; k0 < N; k0 += L) test(min(k0 + l, N - 1));
  }
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    const float e0 = __shfl_xor_sync(0xffffffffu, b0, o), e1 = __shfl_xor_sync(0xffffffffu, b1, o);
    const int k0 = __shfl_xor_sync(0xffffffffu, j0, o), k1 = __shfl_xor_sync(0xffffffffu, j1, o);
    if (k0 >= 0 && (j0 < 0 || e0 < b0 || (e0 == b0 && k0 < j0))) {
      b0 = e0;
      j0 = k0;
    }
    if (k1 >= 0 && (j1 < 0 || e1 < b1 || (e1 == b1 && k1 < j1))) {
      b1 = e1;
      j1 = k1;
    }
  }
  bj[0] = j0;
  bj[1] = j1;
}

// Nearest neighbours of the window nodes [lo, hi) -- a tile at window index 28
// and the 14-node halo its merge states depend on, cut to the level -- into
// s_nb by window index. Called by all THREADS threads; the window holds the
// boxes [lo - 14, hi + 16).
template <int THREADS, int L>
__device__ __forceinline__ void nearest_window(const BoxWindow& w, int lo, int hi, uint16_t* s_nb, uint32_t* status) {
  const int first = lo & ~1, pairs = (hi - first + 1) / 2;
  // whole warps take part (shuffles): the last groups repeat the last pair
  for (int p0 = (threadIdx.x & ~31u) / L; p0 < pairs; p0 += THREADS / L) {
    const int p = min(p0 + (int)(threadIdx.x & 31u) / L, pairs - 1);
    const int i0 = first + 2 * p;
    int bj[2];
    nearest_pair<L>(w, i0, bj);
    if ((threadIdx.x & (L - 1)) != 0) continue;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = i0 + q;
      if (i < lo || i >= hi) continue;
      if (bj[q] < 0) atomicOr(status, kStatusNoNeighbour);
      s_nb[i] = (uint16_t)(bj[q] < 0 ? i : bj[q]);
    }
  }
}

// As many lanes per pair as there are threads for: few nodes per block leave
// a level bound by the latency of the search.
template <int THREADS>
__device__ __forceinline__ void nearest_window_any(const BoxWindow& w, int lo, int hi, uint16_t* s_nb,
                                                   uint32_t* status) {
  const int pairs = (hi - lo + 2) / 2;
  if (pairs * 16 <= THREADS) nearest_window<THREADS, 16>(w, lo, hi, s_nb, status);
  else if (pairs * 8 <= THREADS) nearest_window<THREADS, 8>(w, lo, hi, s_nb, status);
  else if (pairs * 4 <= THREADS) nearest_window<THREADS, 4>(w, lo, hi, s_nb, status);
  else if (pairs * 2 <= THREADS) nearest_window<THREADS, 2>(w, lo, hi, s_nb, status);
  else nearest_window<THREADS, 1>(w, lo, hi, s_nb, status);
}

__device__ __forceinline__ DAabb pair_parent(const DAabb& a, const DAabb& b, uint32_t first_child) {
  DAabb p;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    p.min[ax] = rs_min(b.min[ax], a.min[ax]);
    p.max[ax] = rs_max(b.max[ax], a.max[ax]);
  }
  p.count = -1;
  p.left_first = (int32_t)first_child;
  return p;
}

// ------------------------------------------------------------------ levels in global memory
// A block of THREADS threads takes tiles of two nodes per thread.
template <int THREADS>
struct TileShared {
  static constexpr int kTile = 2 * THREADS;
  static constexpr int kWindow = kTile + 2 * kHalo + 4;
};

// Phase A for the tile [s0, s1) of a block's chunk of the level [begin, end):
// neighbours, then each tile node's neighbour and merge state to nb. Returns
// the thread's count of pair heads.
template <int THREADS>
__device__ uint32_t nn_state_tile(const DAabb* in, uint32_t* nb, uint32_t begin, uint32_t end, uint32_t s0,
                                  uint32_t s1, const BoxWindow& w, uint16_t* s_nb, uint32_t* status) {
  const int len = (int)(s1 - s0);
  const int64_t base = (int64_t)s0 - kHalo;  // node of window index 0
  for (int k = threadIdx.x; k < len + 2 * kHalo + 2; k += THREADS) {
    const int64_t idx = base + k;
    if (idx >= (int64_t)begin && idx < (int64_t)end) {
      const float4* q = reinterpret_cast<const float4*>(in + idx);
      w.set(k, __ldcg(q), __ldcg(q + 1));
    } else {
      w.set_outside(k);
    }
  }
  __syncthreads();
  const int lo = (int)((int64_t)begin > base ? (int64_t)begin - base : 0);
  const int hi = (int)((int64_t)end - base < (int64_t)(len + 2 * kHalo) ? (int64_t)end - base : len + 2 * kHalo);
  nearest_window_any<THREADS>(w, max(lo, kRadius), min(hi, len + kHalo + kRadius), s_nb, status);
  __syncthreads();
  uint32_t heads = 0;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int i = (int)threadIdx.x + q * THREADS;
    if (i >= len) continue;
    const int wi = i + kHalo, j = s_nb[wi];
    const bool mutual = s_nb[j] == wi;
    const uint32_t state = !mutual || j == wi ? 0u : (wi < j ? kPairHead : kPairTail);
    nb[s0 + i] = (uint32_t)(base + j) | state;
    heads += state == kPairHead ? 1u : 0u;
  }
  __syncthreads();
  return heads;
}

// Phase B for the tile [s0, s1): the prefix of the pair heads (carry: heads
// before s0 in the level) and the placement (locb.rs:178-215) from the nb
// words phase A left (heads up to 14 nodes past s1 may belong to the next
// block's chunk). s_word: 2 THREADS + 14 words. Returns the carry for the
// next tile.
template <int THREADS>
__device__ uint32_t place_tile(const DAabb* in, DAabb* out, DAabb* final_nodes, const uint32_t* nb, uint32_t begin,
                               uint32_t end, uint32_t s0, uint32_t s1, uint32_t carry, uint32_t mc, uint32_t* s_word,
                               uint32_t* s_warp, uint32_t* status) {
  const uint32_t span = s1 - s0 + kRadius;
  for (uint32_t k = threadIdx.x; k < span; k += THREADS) {
    const uint32_t idx = s0 + k;
    s_word[k] = idx < end ? __ldcg(nb + idx) : 0u;
  }
  __syncthreads();
  const uint32_t i0 = s0 + 2u * threadIdx.x;
  const uint32_t w0 = i0 < s1 ? s_word[i0 - s0] : 0u, w1 = i0 + 1u < s1 ? s_word[i0 + 1u - s0] : 0u;
  const uint32_t h0 = (w0 & kPairHead) ? 1u : 0u, h1 = (w1 & kPairHead) ? 1u : 0u;
  uint32_t tile_total;
  const uint32_t incl = block_inclusive_scan<THREADS>(h0 + h1, s_warp, &tile_total) + carry;
  const uint32_t unmerged_begin = begin - mc;
  const uint32_t children_begin = end - 2u * mc;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint32_t i = i0 + q;
    if (i >= s1) continue;
    const uint32_t w = q ? w1 : w0;
    const uint32_t merged_i = q ? incl : incl - h1;
    if (w & kPairHead) {
      const uint32_t j = w & kNbMask;
      uint32_t merged_j = merged_i;
      for (uint32_t k = i + 1; k <= j; ++k) merged_j += (s_word[k - s0] & kPairHead) ? 1u : 0u;
      const uint32_t pos = unmerged_begin + j - begin - merged_j;
      const uint32_t fc = children_begin + (merged_i - 1u) * 2u;
      if (j < end && pos < end && fc + 1 < end) {
        const DAabb a = load_aabb_cg(in + i), b = load_aabb_cg(in + j);
        store_aabb(out + pos, pair_parent(a, b, fc));
        store_aabb(final_nodes + fc, a);
        store_aabb(final_nodes + fc + 1, b);
      } else {
        atomicOr(status, kStatusBadIndex);
      }
    } else if (!(w & kPairTail)) {
      const uint32_t pos = unmerged_begin + i - begin - merged_i;
      if (pos < end) store_aabb(out + pos, load_aabb_cg(in + i));
      else atomicOr(status, kStatusBadIndex);
    }
  }
  __syncthreads();
  return carry + tile_total;
}

// The clustering levels of more than p.stop nodes, with a grid barrier after
// each phase.
__global__ void __launch_bounds__(kBlock) k_locb_levels(LocbParams p) {
  using T = TileShared<kBlock>;
  __shared__ float4 s_a[T::kWindow], s_b[T::kWindow];
  __shared__ uint16_t s_nb[T::kWindow];
  __shared__ uint32_t s_word[T::kTile + kRadius];
  __shared__ uint32_t s_warp[kBlock / 32];
  const BoxWindow w{s_a, s_b, T::kWindow / 2};
  const uint32_t node_count = 2u * p.n - 1u;
  uint32_t begin = p.n - 1u, end = node_count;
  int cur = 0;
  const uint32_t G = gridDim.x;
  uint32_t levels = 0;

  while (end - begin > p.stop) {
    const uint32_t m = end - begin;
    const DAabb* in = p.lvl[cur];
    DAabb* out = p.lvl[cur ^ 1];
    const uint32_t chunk = (m + G - 1) / G;
    const uint32_t c0 = min(begin + blockIdx.x * chunk, end);
    const uint32_t c1 = min(c0 + chunk, end);
    uint32_t local = 0;
    for (uint32_t s0 = c0; s0 < c1; s0 += T::kTile)
      local += nn_state_tile<kBlock>(in, p.nb, begin, end, s0, min(s0 + T::kTile, c1), w, s_nb, p.status);
    uint32_t tot;
    block_inclusive_scan<kBlock>(local, s_warp, &tot);
    if (threadIdx.x == 0) p.blocksum[blockIdx.x] = tot;
    if (!grid_sync(p.bar, G, p.status)) return;

    uint32_t pre = 0, all = 0;
    for (uint32_t b = threadIdx.x; b < G; b += kBlock) {
      uint32_t v = __ldcg(p.blocksum + b);
      all += v;
      if (b < blockIdx.x) pre += v;
    }
    uint32_t pre_tot, all_tot;
    block_inclusive_scan<kBlock>(pre, s_warp, &pre_tot);
    block_inclusive_scan<kBlock>(all, s_warp, &all_tot);
    const uint32_t mc = all_tot;
    if (mc == 0) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(p.status, kStatusNoMerge);
      return;
    }
    uint32_t carry = pre_tot;
    for (uint32_t s0 = c0; s0 < c1; s0 += T::kTile)
      carry = place_tile<kBlock>(in, out, p.final_nodes, p.nb, begin, end, s0, min(s0 + T::kTile, c1), carry, mc,
                                 s_word, s_warp, p.status);
    if (!grid_sync(p.bar, G, p.status)) return;
    begin -= mc;
    end -= 2u * mc;
    cur ^= 1;
    ++levels;
  }

  // the rest: k_locb_cluster
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    p.info[0] = levels;
    p.info[1] = begin;
    p.info[2] = end;
    p.info[3] = (uint32_t)cur;
  }
}

// ------------------------------------------------------------------ levels in a cluster's shared memory
constexpr int kClusterThreads = 512;
constexpr uint32_t kClusterCap = 2048;  // nodes per block
constexpr uint32_t kClusterAlone = 256;  // levels of at most so many nodes are block 0's alone
constexpr uint32_t kClusterMinChunk = 64;  // nodes per block at least (a halo of 28 lies in the next block)
constexpr uint32_t kClusterMax = 16;     // blocks of a cluster at most
constexpr int kClusterWindow = (int)kClusterCap + 2 * kHalo + 4;

struct ClusterShared {
  float4 a[2][kClusterWindow], b[2][kClusterWindow];
  uint32_t incl[kClusterCap];  // pair heads up to and with the node, in the block's chunk
  uint32_t sums[kClusterMax];  // pair heads of every block's chunk
  uint32_t warp[kClusterCap / 32];
  uint16_t nb[kClusterWindow];
};
static_assert(TileShared<kClusterThreads>::kWindow <= kClusterWindow, "tiles of the global levels fit the window");
static_assert(TileShared<kClusterThreads>::kTile + kRadius <= (int)kClusterCap, "tile words fit incl");

// Orders shared memory of the cluster's blocks (release / acquire at cluster
// scope).
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same with the blocks' global memory read through L2 (__ldcg).
__device__ __forceinline__ void cluster_barrier() {
  __threadfence();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of this block's shared variable in block `rank` of the cluster.
__device__ __forceinline__ uint32_t remote(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(r)
               : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_remote4(const void* p, uint32_t rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote(p, rank))
               : "memory");
  return v;
}
__device__ __forceinline__ void st_remote4(const void* p, uint32_t rank, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(remote(p, rank)), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}
__device__ __forceinline__ uint32_t ld_remote(const void* p, uint32_t rank) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ void st_remote(const void* p, uint32_t rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(p, rank)), "r"(v) : "memory");
}

// Nodes per block of a level of m nodes: block r has [r chunk, (r + 1) chunk).
__device__ __forceinline__ uint32_t cluster_chunk(uint32_t m, uint32_t blocks) {
  return m <= kClusterAlone ? kClusterAlone : max((m + blocks - 1u) / blocks, kClusterMinChunk);
}

// The levels of at most 32 nodes by one warp, a node per lane: no barriers,
// and the distance of a pair computed once, by its left node. xs: the nodes,
// in index order (scratch afterwards).
__device__ void warp_levels(BoxWindow xs, DAabb* final_nodes, uint32_t begin, uint32_t end, uint32_t* status) {
  constexpr uint32_t all = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, upto = all >> (31u - lane);
  const float inf = __int_as_float(0x7f800000);
  float4 u = xs.a[xs.at(kHalo + (int)lane)], v = xs.b[xs.at(kHalo + (int)lane)];
  while (end - begin > 1u) {
    const uint32_t m = end - begin;
    if (lane >= m) {  // the infinite box never wins (BoxWindow::set_outside)
      u = make_float4(-inf, -inf, -inf, 0.0f);
      v = make_float4(inf, inf, inf, 0.0f);
    }
    SBox x;
    x.mn[0] = u.x; x.mn[1] = u.y; x.mn[2] = u.z;
    x.mx[0] = v.x; x.mx[1] = v.y; x.mx[2] = v.z;
    float right[kRadius];
#pragma unroll
    for (int k = 1; k <= kRadius; ++k) {
      SBox y;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        y.mn[a] = __shfl_down_sync(all, x.mn[a], k);
        y.mx[a] = __shfl_down_sync(all, x.mx[a], k);
      }
      right[k - 1] = union_half_area(x, y);
    }
    float best = 3.40282347e+38f;
    int j = -1;
#pragma unroll
    for (int k = kRadius; k >= 1; --k) {
      const float d = __shfl_up_sync(all, right[k - 1], k);
      if ((int)lane >= k && d < best) {
        best = d;
        j = (int)lane - k;
      }
    }
#pragma unroll
    for (int k = 1; k <= kRadius; ++k) {
      if ((int)lane + k < 32 && right[k - 1] < best) {
        best = right[k - 1];
        j = (int)lane + k;
      }
    }
    if (j < 0) {
      if (lane < m) atomicOr(status, kStatusNoNeighbour);
      j = (int)lane;
    }
    const bool mutual = __shfl_sync(all, j, j) == (int)lane && j != (int)lane && lane < m;
    const uint32_t heads = __ballot_sync(all, mutual && j > (int)lane);
    const uint32_t mc = __popc(heads);
    if (mc == 0u) {
      if (lane == 0u) atomicOr(status, kStatusNoMerge);
      return;
    }
    const uint32_t merged = __popc(heads & upto);
    DAabb a, b;
    a.min[0] = u.x; a.min[1] = u.y; a.min[2] = u.z; a.count = __float_as_int(u.w);
    a.max[0] = v.x; a.max[1] = v.y; a.max[2] = v.z; a.left_first = __float_as_int(v.w);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b.min[k] = __shfl_sync(all, a.min[k], j);
      b.max[k] = __shfl_sync(all, a.max[k], j);
    }
    b.count = __shfl_sync(all, a.count, j);
    b.left_first = __shfl_sync(all, a.left_first, j);
    uint32_t pos = lane - merged;
    if (mutual && j > (int)lane) {
      pos = (uint32_t)j - __popc(heads & (all >> (31u - (uint32_t)j)));
      const uint32_t fc = end - 2u * mc + (merged - 1u) * 2u;
      store_aabb(final_nodes + fc, a);
      store_aabb(final_nodes + fc + 1u, b);
      a = pair_parent(a, b, fc);
    }
    __syncwarp();
    if (lane < m && !(mutual && j < (int)lane)) {
      const int at = xs.at(kHalo + (int)pos);
      xs.a[at] = make_float4(a.min[0], a.min[1], a.min[2], __int_as_float(a.count));
      xs.b[at] = make_float4(a.max[0], a.max[1], a.max[2], __int_as_float(a.left_first));
    }
    __syncwarp();
    u = xs.a[xs.at(kHalo + (int)lane)];
    v = xs.b[xs.at(kHalo + (int)lane)];
    begin -= mc;
    end -= 2u * mc;
  }
  if (lane == 0u) {
    float4* out = reinterpret_cast<float4*>(final_nodes + begin);
    out[0] = u;
    out[1] = v;
  }
}

// The levels of at most blocks * kClusterCap nodes [begin, end), read from lvl
// in global memory, by a cluster of `blocks` blocks (this one is `rank`):
// the level stays in the blocks' shared memory, chunk by chunk. Every loop
// bound is computed from values all blocks have alike, so each barrier is
// reached by all of them; a block that has left at kClusterAlone nodes is not
// accessed any more. What bounds a level here is latency: two cluster
// barriers (1,200-1,600 cycles each), a remote read for the halos and the
// search with few nodes per thread (up to sixteen lanes share a pair). It
// replaces one block of 1024 threads from 2048 nodes on, and grid barriers
// above. 6,400 triangles 183 -> 103 us, 1M: the 38 levels below
// 32,768 nodes 146 us (118 us went to the last 25 of them alone).
__device__ void cluster_levels(ClusterShared& s, const DAabb* lvl, DAabb* final_nodes, uint32_t begin, uint32_t end,
                               uint32_t rank, uint32_t blocks, uint32_t* status) {
  constexpr int T = kClusterThreads;
  const uint32_t tid = threadIdx.x;
  uint32_t chunk = cluster_chunk(end - begin, blocks);
  int cur = 0;
  {
    const uint32_t m = end - begin, c0 = min(rank * chunk, m), len = min(chunk, m - c0);
    const BoxWindow w{s.a[0], s.b[0], kClusterWindow / 2};
    for (uint32_t k = tid; k < len; k += T) {
      const float4* q = reinterpret_cast<const float4*>(lvl + begin + c0 + k);
      w.set(kHalo + (int)k, __ldcg(q), __ldcg(q + 1));
    }
  }
  if (end - begin > kClusterAlone) cluster_sync();
  else __syncthreads();
  while (end - begin > 32u) {
    const uint32_t m = end - begin;
    const bool alone = m <= kClusterAlone;
    if (alone && rank != 0u) return;
    const uint32_t c0 = min(rank * chunk, m), len = min(chunk, m - c0);
    const BoxWindow w{s.a[cur], s.b[cur], kClusterWindow / 2};
    // halos: the last 28 nodes of the block before, the first 28 of the next
    if (len && tid < 2u * kHalo + 2u) {
      const bool left = tid < (uint32_t)kHalo;
      const uint32_t k = left ? tid : tid - kHalo;
      const int wi = left ? (int)k : (int)(kHalo + len + k);
      const bool there = left ? c0 > 0u : (k < (uint32_t)kHalo && c0 + len + k < m);
      if (there) {
        const int at = w.at(left ? (int)(chunk + k) : (int)(kHalo + k));  // chunk - 28 + k there, + 28
        const uint32_t from = left ? rank - 1u : rank + 1u;
        w.set(wi, ld_remote4(w.a + at, from), ld_remote4(w.b + at, from));
      } else {
        w.set_outside(wi);
      }
    }
    __syncthreads();
    if (len) {
      const int lo = c0 > 0u ? kRadius : kHalo;
      const int hi = (int)min(len + kHalo + kRadius, m - c0 + kHalo);
      nearest_window_any<T>(w, lo, hi, s.nb, status);
    }
    __syncthreads();
    // merge flags and their prefix in the chunk: thread t has the nodes
    // t + q T; a warp's flags of one q are a ballot
    constexpr int Q = (int)kClusterCap / T;
    const uint32_t lane = tid & 31u, warp = tid >> 5, per = (len + T - 1u) / T;
    int nbr[Q];         // neighbour of a pair's head, -1: unmerged, -2: a pair's tail or no node
    uint32_t flags[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (q >= (int)per) break;
      const uint32_t i = tid + (uint32_t)(q * T);
      nbr[q] = -2;
      if (i < len) {
        const int wi = (int)i + kHalo, j = s.nb[wi];
        const bool mutual = j != wi && s.nb[j] == wi;
        nbr[q] = !mutual ? -1 : (j > wi ? j : -2);
      }
      flags[q] = __ballot_sync(0xffffffffu, nbr[q] >= 0);
      if (lane == 0u) s.warp[q * (T / 32) + warp] = __popc(flags[q]);
    }
    __syncthreads();
    uint32_t merged[Q];  // pair heads up to and with the node
    uint32_t total = 0;
    {
      const uint32_t n = per * (T / 32);
      uint32_t v0 = lane < n ? s.warp[lane] : 0u, v1 = lane + 32u < n ? s.warp[lane + 32u] : 0u;
      const uint32_t c0w = v0, c1w = v1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u0 = __shfl_up_sync(0xffffffffu, v0, o);
        const uint32_t u1 = n > 32u ? __shfl_up_sync(0xffffffffu, v1, o) : 0u;
        if (lane >= (uint32_t)o) {
          v0 += u0;
          v1 += u1;
        }
      }
      const uint32_t t0 = __shfl_sync(0xffffffffu, v0, 31);
      total = t0 + (n > 32u ? __shfl_sync(0xffffffffu, v1, 31) : 0u);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (q >= (int)per) break;
        const int e = (q * (T / 32) + (int)warp) & 31;
        const uint32_t before = q * (T / 32) < 32 ? __shfl_sync(0xffffffffu, v0 - c0w, e)
                                                  : t0 + __shfl_sync(0xffffffffu, v1 - c1w, e);
        merged[q] = before + __popc(flags[q] & (0xffffffffu >> (31u - lane)));
        const uint32_t i = tid + (uint32_t)(q * T);
        if (i < len) s.incl[i] = merged[q];
      }
    }
    uint32_t mc = total, pre = 0;
    if (alone) {
      __syncthreads();
    } else {
      if (tid < blocks) st_remote(s.sums + rank, tid, total);
      cluster_sync();
      mc = 0;
      for (uint32_t b = 0; b < blocks; ++b) {
        const uint32_t v = s.sums[b];
        mc += v;
        if (b < rank) pre += v;
      }
    }
    if (mc == 0u) {  // the same in every block
      if (rank == 0u && tid == 0u) atomicOr(status, kStatusNoMerge);
      return;
    }
    // parents of merged pairs and unmerged nodes to the next level, merged
    // pairs' children to the final node array (locb.rs:178-215)
    const uint32_t next_m = m - mc, next_chunk = cluster_chunk(next_m, blocks);
    // block of a position: positions are below 2^15, so (pos + 0.5) / chunk
    // is further from an integer than the float arithmetic's error
    const float chunk_rcp = 1.0f / (float)next_chunk;
    const uint32_t children_begin = end - 2u * mc;
    const BoxWindow nw{s.a[cur ^ 1], s.b[cur ^ 1], kClusterWindow / 2};
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (q >= (int)per) break;
      const int j = nbr[q];
      if (j == -2) continue;
      const uint32_t i = tid + (uint32_t)(q * T), merged_i = pre + merged[q];
      const DAabb x = w.node((int)i + kHalo);
      uint32_t pos;
      DAabb out = x;
      if (j >= 0) {
        const uint32_t jr = (uint32_t)(j - kHalo);
        const uint32_t merged_j =
            jr < len ? pre + s.incl[jr] : pre + total + ld_remote(s.incl + (jr - len), rank + 1u);
        pos = c0 + jr - merged_j;
        const uint32_t fc = children_begin + (merged_i - 1u) * 2u;
        const DAabb y = w.node(j);
        out = pair_parent(x, y, fc);
        if (fc + 1u < end) {
          store_aabb(final_nodes + fc, x);
          store_aabb(final_nodes + fc + 1u, y);
        } else {
          atomicOr(status, kStatusBadIndex);
        }
      } else {
        pos = c0 + i - merged_i;
      }
      if (pos >= next_m) {
        atomicOr(status, kStatusBadIndex);
        continue;
      }
      const float4 u = make_float4(out.min[0], out.min[1], out.min[2], __int_as_float(out.count));
      const float4 v = make_float4(out.max[0], out.max[1], out.max[2], __int_as_float(out.left_first));
      const uint32_t owner = alone ? 0u : (uint32_t)(((float)pos + 0.5f) * chunk_rcp);
      const int at = nw.at((int)(pos - owner * next_chunk) + kHalo);
      if (owner == rank) {
        nw.a[at] = u;
        nw.b[at] = v;
      } else {
        st_remote4(nw.a + at, owner, u);
        st_remote4(nw.b + at, owner, v);
      }
    }
    if (alone) __syncthreads();
    else cluster_sync();
    begin -= mc;
    end -= 2u * mc;
    chunk = next_chunk;
    cur ^= 1;
  }
  if (rank == 0u && tid < 32u)
    warp_levels(BoxWindow{s.a[cur], s.b[cur], kClusterWindow / 2}, final_nodes, begin, end, status);
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_blocks() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// One cluster: the levels k_locb_levels left (p.info) or, for builds with no
// such level, all of them.
__global__ void __launch_bounds__(kClusterThreads) k_locb_cluster(LocbParams p, bool from_info, uint32_t begin0,
                                                                  uint32_t end0) {
  extern __shared__ __align__(16) unsigned char cluster_smem[];
  ClusterShared& s = *reinterpret_cast<ClusterShared*>(cluster_smem);
  const uint32_t begin = from_info ? __ldcg(p.info + 1) : begin0;
  const uint32_t end = from_info ? __ldcg(p.info + 2) : end0;
  const uint32_t cur = from_info ? __ldcg(p.info + 3) : 0u;
  const uint32_t blocks = cluster_blocks();
  if (end <= begin || end - begin > blocks * kClusterCap || end > 2u * p.n - 1u || cur > 1u || blocks > kClusterMax) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(p.status, kStatusBadIndex);
    return;  // the same in every block
  }
  cluster_levels(s, p.lvl[cur], p.final_nodes, begin, end, cluster_rank(), blocks, p.status);
}

// Leaves: sorted boxes + 1e-4, count 1, left_first = i (locb.rs:289-294).
__global__ void __launch_bounds__(kBlock)
    k_locb_leaves(const DAabb* __restrict__ aabbs, const uint32_t* __restrict__ sorted, uint32_t n,
                  DAabb* __restrict__ lvl) {
  uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= n) return;
  DAabb b = load_aabb(aabbs + __ldg(sorted + i));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.min[a] = b.min[a] - 0.0001f;
    b.max[a] = b.max[a] + 0.0001f;
  }
  b.count = 1;
  b.left_first = (int32_t)i;
  store_aabb(lvl + (n - 1u) + i, b);
}

// n <= 2: one root leaf holding the world box (locb.rs:258-269).
__global__ void k_locb_single(const DAabb* world, uint32_t n, DAabb* nodes, uint32_t* indices) {
  if (threadIdx.x == 0) {
    DAabb w = *world;
    w.count = (int32_t)n;
    w.left_first = 0;
    store_aabb(nodes, w);
  }
  if (threadIdx.x < n) indices[threadIdx.x] = threadIdx.x;
}


// ---------------------------------------------------------------- many meshes
// A cluster of blocks per mesh clusters the mesh's own node range of a
// concatenated forest. Mesh m owns primitives [off_m, off_m + n_m) and nodes
// [2 off_m - m, 2 off_m - m + 2 n_m - 1); the placement arithmetic of a level
// depends only on differences of indices, so every node, left_first and
// leaf offset comes out as the single-mesh build's shifted by the mesh's
// offsets.
struct SegParams {
  DAabb* lvl[2];
  DAabb* final_nodes;
  uint32_t* nb;
  const uint32_t* prim_off;   // mesh_count + 1
  const uint32_t* order;      // meshes in processing order (largest first)
  const DAabb* worlds;        // per-mesh union_of_list boxes
  uint32_t* indices;          // sorted primitive indices (global); identity for n <= 2
  uint32_t* status;
  uint32_t mesh_count;
};

// Meshes order[first, last), one at a time per cluster (of one block or
// more; sums: a word per block): levels too large for the cluster's shared
// memory in global memory with cluster barriers, the rest by cluster_levels.
// Every block of a cluster runs the same mesh sequence and the same level
// count (all loop bounds are computed from values every block reads
// identically), so each barrier is reached by all of them; nothing waits on
// another cluster. Blocks that are done with a mesh early (kClusterAlone)
// wait for block 0 at the next mesh's first barrier.
__global__ void __launch_bounds__(kClusterThreads) k_locb_forest(SegParams p, uint32_t* cluster_sums, uint32_t first,
                                                                 uint32_t last) {
  extern __shared__ __align__(16) unsigned char cluster_smem[];
  ClusterShared& s = *reinterpret_cast<ClusterShared*>(cluster_smem);
  constexpr int T = kClusterThreads;
  using Tile = TileShared<T>;
  const uint32_t blocks = cluster_blocks(), rank = cluster_rank();
  const uint32_t cid = blockIdx.x / blocks, ncl = gridDim.x / blocks;
  uint32_t* sums = cluster_sums + (size_t)cid * blocks;
  for (uint32_t q = first + cid; q < last; q += ncl) {
    const uint32_t m = p.order[q];
    const uint32_t off = p.prim_off[m], n = p.prim_off[m + 1] - off;
    if (n == 0) continue;
    const uint32_t nbase = 2u * off - m;
    if (n <= 2) {
      if (rank == 0 && threadIdx.x == 0) {
        DAabb w = p.worlds[m];
        w.count = (int32_t)n;
        w.left_first = (int32_t)off;
        store_aabb(p.final_nodes + nbase, w);
      }
      if (rank == 0 && threadIdx.x < n) p.indices[off + threadIdx.x] = off + threadIdx.x;
      continue;
    }
    uint32_t begin = nbase + n - 1u, end = nbase + 2u * n - 1u;
    int cur = 0;
    bool ok = true;
    cluster_barrier();  // block 0 is done with the mesh before
    while (end - begin > blocks * kClusterCap) {
      const BoxWindow w{s.a[0], s.b[0], Tile::kWindow / 2};
      const uint32_t count = end - begin;
      const DAabb* in = p.lvl[cur];
      DAabb* out = p.lvl[cur ^ 1];
      const uint32_t chunk = (count + blocks - 1) / blocks;
      const uint32_t c0 = min(begin + rank * chunk, end);
      const uint32_t c1 = min(c0 + chunk, end);
      uint32_t local = 0;
      for (uint32_t s0 = c0; s0 < c1; s0 += Tile::kTile)
        local += nn_state_tile<T>(in, p.nb, begin, end, s0, min(s0 + Tile::kTile, c1), w, s.nb, p.status);
      uint32_t tot;
      block_inclusive_scan<T>(local, s.warp, &tot);
      if (threadIdx.x == 0) sums[rank] = tot;
      cluster_barrier();
      uint32_t pre = 0, mc = 0;
      for (uint32_t b = 0; b < blocks; ++b) {
        const uint32_t v = __ldcg(sums + b);
        mc += v;
        if (b < rank) pre += v;
      }
      if (mc == 0) {  // same value in every block of the cluster
        if (rank == 0 && threadIdx.x == 0) atomicOr(p.status, kStatusNoMerge);
        ok = false;
        break;
      }
      uint32_t carry = pre;
      for (uint32_t s0 = c0; s0 < c1; s0 += Tile::kTile)
        carry = place_tile<T>(in, out, p.final_nodes, p.nb, begin, end, s0, min(s0 + Tile::kTile, c1), carry, mc,
                              s.incl, s.warp, p.status);
      cluster_barrier();
      begin -= mc;
      end -= 2u * mc;
      cur ^= 1;
    }
    if (ok) cluster_levels(s, p.lvl[cur], p.final_nodes, begin, end, rank, blocks, p.status);
  }
  cluster_barrier();  // no block leaves while another may still reach into it
}

// Leaves of every mesh: sorted position k of mesh m (off_m <= k < off_m + n_m)
// becomes node 2 off_m - m + n_m - 1 + (k - off_m) with the primitive's box
// + 1e-4, count 1, left_first = k.
__global__ void __launch_bounds__(kBlock)
    k_locb_segment_leaves(const DAabb* __restrict__ aabbs, const uint32_t* __restrict__ sorted,
                          const uint32_t* __restrict__ prim_off, uint32_t mesh_count, uint32_t total,
                          DAabb* __restrict__ lvl) {
  const uint32_t k = blockIdx.x * kBlock + threadIdx.x;
  if (k >= total) return;
  uint32_t lo = 0, hi = mesh_count;  // mesh with prim_off[m] <= k < prim_off[m + 1]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(prim_off + mid) <= k) lo = mid;
    else hi = mid;
  }
  const uint32_t m = lo, off = __ldg(prim_off + m), n = __ldg(prim_off + m + 1) - off;
  if (n <= 2) return;
  DAabb b = load_aabb(aabbs + __ldg(sorted + k));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.min[a] = b.min[a] - 0.0001f;
    b.max[a] = b.max[a] + 0.0001f;
  }
  b.count = 1;
  b.left_first = (int32_t)k;
  store_aabb(lvl + (2u * off - m) + (n - 1u) + (k - off), b);
}

// Launches `clusters` clusters of `blocks` blocks with the cluster kernels'
// shared memory.
template <class K, class... Args>
cudaError_t launch_cluster(K kern, unsigned clusters, unsigned blocks, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * blocks);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = sizeof(ClusterShared);
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = blocks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Blocks of the largest cluster the current device can hold (16 where it is
// allowed, else the portable 8); sets the kernels' attributes on its first use.
cudaError_t cluster_size(unsigned* blocks) {
  static PerDevice<unsigned> sizes;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e) return e;
  return sizes.get(dev, blocks, [](unsigned* size) {
    for (auto k : {reinterpret_cast<const void*>(k_locb_cluster), reinterpret_cast<const void*>(k_locb_forest)}) {
      cudaError_t err =
          cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterShared));
      if (err) return err;
    }
    *size = 8;
    if (cudaFuncSetAttribute(k_locb_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return cudaSuccess;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterMax);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterShared);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kClusterMax;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_locb_cluster, &cfg) == cudaSuccess && n > 0) *size = kClusterMax;
    else cudaGetLastError();
    return cudaSuccess;
  });
}

}  // namespace

ResultCode build_locb(const DAabb* aabbs, const float4* centers, size_t n_, cudaStream_t s, BuildOutput* out) {
  if (n_ == 0) return NoPrimitives;
  if (n_ >= (1u << 30)) return InvalidArgument;
  const uint32_t n = (uint32_t)n_;
  const uint32_t node_count = n <= 2 ? 1u : 2u * n - 1u;
  cudaError_t e;
  DAabb* nodes = nullptr;
  uint32_t* indices = nullptr;
  if ((e = device_alloc(&nodes, node_count, s)) != cudaSuccess) return cuda_rc(e);
  if ((e = device_alloc(&indices, n, s)) != cudaSuccess) {
    pool_free(nodes, s);
    return cuda_rc(e);
  }
  auto fail = [&](ResultCode rc) {
    pool_free(nodes, s);
    pool_free(indices, s);
    return rc;
  };
  int dev = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_locb_levels, kBlock, 0);
  if (per_sm < 1) return fail(DeviceError);
  // Up to a million primitives at most 3 blocks per SM: fewer blocks make the
  // grid barriers between clustering levels cheaper; above, a level's work
  // counts for more. 3 against 4 blocks (all that fit), us: 200k 812 / 822, 1M
  // 1,414 / 1,414, 4M 3,860 / 3,767, 10M 10,921 / 10,481; 2 blocks: 812, 1,444,
  // 4,116, 12,220.
  if (per_sm > 3 && n <= 1000000u) per_sm = 3;
  unsigned grid = (unsigned)(sm_count() * per_sm);
  const unsigned useful = (unsigned)((n + kBlock - 1) / kBlock);
  if (grid > useful) grid = useful;
  if (grid < 1) grid = 1;
  ScratchPack scratch;
  DAabb *world, *lvl0 = nullptr, *lvl1 = nullptr;
  uint32_t *acc, *status, *keys = nullptr, *nb = nullptr, *blocksum = nullptr;
  char* sort_temp = nullptr;
  constexpr size_t kBarWords = (sizeof(GridBarrier) + 3) / 4;
  const size_t sort_bytes = radix_sort_temp_bytes(n);
  scratch.add(&world, 1);
  scratch.add(&acc, kBoundsWords);
  scratch.add(&status, 8 + kBarWords);  // status, info, barrier
  if (n > 2) {
    scratch.add(&keys, n);
    scratch.add(&sort_temp, sort_bytes);
    scratch.add(&lvl0, node_count);
    scratch.add(&lvl1, node_count);
    scratch.add(&nb, node_count);
    scratch.add(&blocksum, grid);
  }
  if ((e = scratch.alloc(s)) || (e = cudaMemsetAsync(status, 0, (8 + kBarWords) * 4, s))) return fail(cuda_rc(e));
  if ((e = launch_world_bounds(aabbs, n, world, acc, s))) return fail(cuda_rc(e));
  if (n <= 2) {
    k_locb_single<<<1, 32, 0, s>>>(world, n, nodes, indices);
    if ((e = cudaGetLastError()) || (e = cudaStreamSynchronize(s))) return fail(cuda_rc(e));
    out->nodes = nodes;
    out->indices = indices;
    out->node_count = 1;
    return Ok;
  }
  if ((e = launch_morton(centers, n, world, keys, indices, s))) return fail(cuda_rc(e));
  if ((e = radix_sort_pairs(keys, indices, n, 30, sort_temp, sort_bytes, status, s))) return fail(cuda_rc(e));
  k_locb_leaves<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(aabbs, indices, n, lvl0);
  if ((e = cudaGetLastError())) return fail(cuda_rc(e));

  LocbParams p;
  p.lvl[0] = lvl0;
  p.lvl[1] = lvl1;
  p.final_nodes = nodes;
  p.nb = nb;
  p.blocksum = blocksum;
  p.bar = reinterpret_cast<GridBarrier*>(status + 8);
  p.status = status;
  p.info = status + 4;
  p.n = n;
  unsigned blocks = 0;
  if ((e = cluster_size(&blocks))) return fail(cuda_rc(e));
  p.stop = blocks * kClusterCap;
  const bool wide = n > p.stop;  // larger levels in the cooperative launch
  if (wide) {
    void* args[] = {&p};
    if ((e = cudaLaunchCooperativeKernel((void*)k_locb_levels, dim3(grid), dim3(kBlock), args, 0, s)))
      return fail(cuda_rc(e));
  }
  if ((e = launch_cluster(k_locb_cluster, 1, blocks, s, p, wide, n - 1u, node_count))) return fail(cuda_rc(e));
  uint32_t h_status = 0;
  if ((e = cudaMemcpyAsync(&h_status, status, 4, cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s)))
    return fail(cuda_rc(e));
  if (h_status & kStatusTimeout) return fail(Timeout);
  if (h_status) return fail(Error);
  out->nodes = nodes;
  out->indices = indices;
  out->node_count = node_count;
  return Ok;
}

}  // namespace rtbvh

namespace rtbvh {

cudaError_t launch_locb_segments(const DAabb* aabbs, const uint32_t* sorted, uint32_t* indices,
                                 const uint32_t* prim_off, const uint32_t* order, const DAabb* worlds,
                                 uint32_t mesh_count, uint32_t total_prims, DAabb* lvl0, DAabb* lvl1,
                                 DAabb* final_nodes, uint32_t* nb, uint32_t* status, unsigned blocks,
                                 uint32_t big_count, uint32_t* cluster_sums, unsigned clusters, unsigned cluster_blocks,
                                 cudaStream_t s, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
  if (total_prims == 0 || mesh_count == 0) return cudaSuccess;
  if (big_count > mesh_count || (big_count > 0 && (clusters == 0 || cluster_blocks == 0 ||
                                                   cluster_blocks > kSegCluster || cluster_sums == nullptr)))
    return cudaErrorInvalidValue;
  cudaError_t e;
  k_locb_segment_leaves<<<(total_prims + kBlock - 1) / kBlock, kBlock, 0, s>>>(aabbs, sorted, prim_off, mesh_count,
                                                                                total_prims, lvl0);
  SegParams p;
  p.lvl[0] = lvl0;
  p.lvl[1] = lvl1;
  p.final_nodes = final_nodes;
  p.nb = nb;
  p.prim_off = prim_off;
  p.order = order;
  p.worlds = worlds;
  p.indices = indices;
  p.status = status;
  p.mesh_count = mesh_count;
  // small meshes (one block each) on the side stream, concurrently with the
  // clusters of the large ones; the two sets of meshes share no memory
  unsigned largest = 0;
  if ((e = cluster_size(&largest))) return e;  // sets the kernel's attributes
  const bool fork_side = side != nullptr && big_count > 0 && big_count < mesh_count;
  cudaStream_t small_s = s;
  if (fork_side) {
    if ((e = cudaEventRecord(fork, s)) || (e = cudaStreamWaitEvent(side, fork, 0))) return e;
    small_s = side;
  }
  if (big_count > 0 &&
      (e = launch_cluster(k_locb_forest, clusters, cluster_blocks, s, p, cluster_sums, 0u, big_count)))
    return e;
  if (big_count < mesh_count) {
    const unsigned nb_small = std::min<unsigned>(blocks, mesh_count - big_count);
    // single blocks use no sums of other blocks: any word does
    if ((e = launch_cluster(k_locb_forest, nb_small, 1, small_s, p, cluster_sums + (size_t)kSegCluster * clusters,
                            big_count, mesh_count)))
      return e;
  }
  if (fork_side) {
    if ((e = cudaEventRecord(join, side)) || (e = cudaStreamWaitEvent(s, join, 0))) return e;
  }
  return cudaSuccess;
}

}  // namespace rtbvh
