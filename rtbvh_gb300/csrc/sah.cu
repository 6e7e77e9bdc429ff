// Binned SAH build (src/builders/binned_sah.rs) on the GPU, breadth first.
//
// The reference runs one task per node (BinnedSahBuildTask::run,
// binned_sah.rs:132-282) from a depth-first work stack. Here the whole build
// is one cooperative launch (k_sah_build) that walks the tree level by
// level; the phases of a level are separated by grid barriers (bounded
// waits), so no host round trip or relaunch happens between levels:
//
//   large tasks (more than sub_max primitives): the grid bins 2048-primitive
//     chunks into per-task global bins (runs of primitives in one bin merged
//     in registers, then ordered-int atomics), one warp per task decides the
//     split, and a chunked stable partition (decoupled look-back over the
//     chunks of a task, bounded waits) scatters the primitive indices;
//   then a scan over the level's tasks numbers the children (breadth-first,
//     deterministic) and builds the next level's task list. Children of at
//     most sub_max primitives are not split level by level: they go to a
//     subtree list. sub_max = n / 2048 clamped to [32, kWarpMax], so a small
//     build keeps enough subtrees to fill the GPU. (It also decides the node
//     numbering: breadth first above it.)
//
// After the last level, k_sub_build builds every listed subtree depth first,
// one warp per subtree (bins in shared memory, the warp-parallel decision,
// ballot partition), large ones in two launches (kMid); what is left, subtrees of at most kSmall primitives, is
// built by k_sub_small, one lane per primitive and several subtrees per warp.
// Neither has grid-wide phases. The node pair of a split at primitive position
// m goes to scratch slots 2(m-1), 2(m-1)+1 -- split positions are distinct
// across the whole tree -- and a scan over the positions places the pairs after
// the breadth-first part in position order, so the numbering stays
// deterministic and gap-free.
//
// The split arithmetic is the reference's: node box + 1e-4; 16 bins per axis
// with bin = min(15, max(c * (16/diag) + off, 0) as usize) (no FMA); the
// right/left cost sweeps of find_split (empty bins give NaN costs that never
// win); axis choice with strict '>'; the max_split_cost test; the
// longest-axis fallback at 2/5 of the primitives; child boxes from the bins
// (the left one over bins [0, best_splits[axis].count), a reference quirk);
// a leaf box gets the 1e-4 offset a second time. Bin contents are exact, so
// every split equals the reference's. The partition is stable where the
// reference's Lomuto partition (src/utils.rs:74-96) is not: leaves hold the
// same primitive sets, possibly in a different order.
#include "lib_internal.h"

namespace rtbvh {

namespace {

constexpr int kBins = 16;
constexpr uint32_t kMaxDepth = 64;
constexpr float kTraversalCost = 1.0f;
constexpr int kChunk = 2048;
constexpr int kLargeBlock = 256;
constexpr uint32_t kWarpMax = 1024;  // largest subtree
constexpr uint32_t kTaskWarp = 64;  // largest task of k_sah_build's lists that one warp does
constexpr uint32_t kCoopMaxPrims = 1u << 21;      // larger builds launch the phases separately
constexpr int kBinWords = 8;  // ordered min xyz, ordered max xyz, count, pad
constexpr int kTaskBinWords = 3 * kBins * kBinWords;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1u;
constexpr float kF32Max = 3.40282347e+38f;

struct Task {
  uint32_t node, begin, end, depth;
};

struct Decision {
  uint32_t split, axis, split_index, n_left;
  float lbox[6];
  float rbox[6];
  uint32_t pad[4];
};
static_assert(sizeof(Decision) == 80, "Decision layout");

struct Counters {
  uint32_t large;       // tasks in the current large list
  uint32_t next_large, next_sub;  // large tasks and subtrees of the level numbered by one block
  uint32_t big[2];      // k_sah_build: whether the list of an even / odd level has tasks above kChunk
  uint32_t sub;         // subtree tasks listed so far (all levels)
  uint32_t node_count;  // nodes of the breadth-first part so far
  uint32_t chunks;      // chunks of the current large list
  uint32_t status;
  uint32_t ticket;      // chunk ticket of the partition kernel
  uint32_t sub_head;    // next subtree a warp of k_sub_build takes
  uint32_t sub_splits;  // splits inside the subtrees (the scan's total)
  uint32_t tiny;        // entries of the small-subtree list
  uint32_t tiny_head;   // next ones a warp of k_sub_small takes
  uint32_t mid, mid_head;  // the same for the list of k_sub_build's second launch
};

struct BinMap {
  float c2b[3], off[3];
};

// binned_sah.rs:146-147
__device__ __forceinline__ BinMap make_binmap(const float mn[3], const float mx[3]) {
  BinMap m;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float inv = 1.0f / (mx[a] - mn[a]);
    m.c2b[a] = inv * (float)kBins;
    m.off[a] = (-mn[a]) * m.c2b[a];
  }
  return m;
}

// compute_bin_index (binned_sah.rs:119-128): min(15, max(f, 0) as usize).
__device__ __forceinline__ uint32_t bin_of(float c, float c2b, float off) {
  float f = c * c2b + off;
  if (f >= 15.0f) return 15u;
  if (f > 0.0f) return (uint32_t)f;
  return 0u;
}

__device__ __forceinline__ float ha6(const float mn[3], const float mx[3]) {
  return half_area(mn[0], mn[1], mn[2], mx[0], mx[1], mx[2]);
}

// A task's bins as ordered keys (kTaskBinWords words in shared memory).
struct BinsView {
  const uint32_t* w;
};

// One bin (or a union of bins) as ordered keys (float_to_ordered). Bin
// bounds are never NaN (triangle boxes grow with Vec3::min/max, which ignore
// NaN, from the empty box), and on non-NaN floats the unsigned min/max of the
// keys is Vec3::min/max (-0 below +0); it is commutative and associative and
// counts are integers, so a union over any grouping of the bins equals the
// reference's sequential Aabb::grow_bb bit for bit.
struct BinKey {
  uint32_t mn[3], mx[3];
  uint32_t cnt;
};

__device__ __forceinline__ BinKey load_bin(const BinsView& B, int a, int i) {
  const uint32_t* w = B.w + (a * kBins + i) * kBinWords;
  BinKey v;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    v.mn[k] = w[k];
    v.mx[k] = w[3 + k];
  }
  v.cnt = w[6];
  return v;
}

__device__ __forceinline__ void bin_union(BinKey& x, const BinKey& y) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x.mn[k] = min(x.mn[k], y.mn[k]);
    x.mx[k] = max(x.mx[k], y.mx[k]);
  }
  x.cnt += y.cnt;
}

__device__ __forceinline__ BinKey shfl_bin(const BinKey& v, int delta, bool up) {
  BinKey r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.mn[k] = up ? __shfl_up_sync(0xffffffffu, v.mn[k], delta, 16) : __shfl_down_sync(0xffffffffu, v.mn[k], delta, 16);
    r.mx[k] = up ? __shfl_up_sync(0xffffffffu, v.mx[k], delta, 16) : __shfl_down_sync(0xffffffffu, v.mx[k], delta, 16);
  }
  r.cnt = up ? __shfl_up_sync(0xffffffffu, v.cnt, delta, 16) : __shfl_down_sync(0xffffffffu, v.cnt, delta, 16);
  return r;
}

// A union of bins decoded to floats.
struct BinVal {
  float mn[3], mx[3];
  uint32_t cnt;
};

__device__ __forceinline__ BinVal decode_bin(const BinKey& k) {
  BinVal v;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    v.mn[q] = ordered_to_float(k.mn[q]);
    v.mx[q] = ordered_to_float(k.mx[q]);
  }
  v.cnt = k.cnt;
  return v;
}

// The sweeps of find_split (binned_sah.rs:80-114) for one axis, bin i =
// lane & 15 of a 16-lane segment: pre = bins [0, i], suf = bins [i, 16).
struct AxisScan {
  BinVal pre, suf;
  float best_cost;
  uint32_t best_count;
};

__device__ __forceinline__ AxisScan scan_axis(const BinsView& B, int a, int i) {
  const BinKey b = load_bin(B, a, i);
  BinKey pre = b, suf = b;
#pragma unroll
  for (int d = 1; d < kBins; d <<= 1) {
    const BinKey lo = shfl_bin(pre, d, true);
    const BinKey hi = shfl_bin(suf, d, false);
    if (i >= d) bin_union(pre, lo);
    if (i + d < kBins) bin_union(suf, hi);
  }
  // both sweeps start from Aabb::empty()
  const uint32_t emn = float_to_ordered(1e34f), emx = float_to_ordered(-1e34f);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    pre.mn[k] = min(pre.mn[k], emn);
    pre.mx[k] = max(pre.mx[k], emx);
    suf.mn[k] = min(suf.mn[k], emn);
    suf.mx[k] = max(suf.mx[k], emx);
  }
  AxisScan r;
  r.pre = decode_bin(pre);
  r.suf = decode_bin(suf);
  // right_cost[i] (i >= 1) and the left sweep's cost at i (i <= 14)
  const float rc = ha6(r.suf.mn, r.suf.mx) * (float)r.suf.cnt;
  const float rc_next = __shfl_down_sync(0xffffffffu, rc, 1, 16);
  const float cost = ha6(r.pre.mn, r.pre.mx) * (float)r.pre.cnt + rc_next;
  // first minimum over i in [0, 15) of the costs below f32::MAX (strict '<'
  // from f32::MAX in ascending order; NaN costs of empty sides never win)
  bool valid = i < kBins - 1 && cost < kF32Max;
  float c = cost;
  uint32_t idx = valid ? (uint32_t)i : (uint32_t)kBins;
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) {
    const float oc = __shfl_xor_sync(0xffffffffu, c, d, 16);
    const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, d, 16);
    const bool ov = oi < (uint32_t)kBins;
    if (ov && (!valid || oc < c || (oc == c && oi < idx))) {
      c = oc;
      idx = oi;
      valid = true;
    }
  }
  r.best_cost = valid ? c : kF32Max;
  r.best_count = valid ? idx + 1u : (uint32_t)kBins;
  return r;
}

// Value of field f of the scan of `axis` at bin j, fetched from the lane
// holding it (A: axes 0 / 1 in lanes 0-15 / 16-31, B: axis 2 in lanes 0-15).
__device__ __forceinline__ float fetch_f(const AxisScan& A, const AxisScan& Bx, int axis, int j, bool pre, int f) {
  const BinVal& va = pre ? A.pre : A.suf;
  const BinVal& vb = pre ? Bx.pre : Bx.suf;
  const float* fa = f < 3 ? va.mn : va.mx;
  const float* fb = f < 3 ? vb.mn : vb.mx;
  const int k = f % 3;
  const float v = axis == 2 ? fb[k] : fa[k];
  return __shfl_sync(0xffffffffu, v, axis == 1 ? 16 + j : j);
}
__device__ __forceinline__ uint32_t fetch_cnt(const AxisScan& A, const AxisScan& Bx, int axis, int j) {
  const uint32_t v = axis == 2 ? Bx.pre.cnt : A.pre.cnt;
  return __shfl_sync(0xffffffffu, v, axis == 1 ? 16 + j : j);
}

// The split decision of BinnedSahBuildTask::run after binning
// (binned_sah.rs:174-247, find_split at :80-114), evaluated by a whole warp
// (every lane returns the same decision). `box` is the node box with its
// first 1e-4 offset.
__device__ void sah_decide_warp(const BinsView& B, const float bmn[3], const float bmx[3], uint32_t ws,
                                uint32_t max_leaf, Decision& d) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  const AxisScan A = scan_axis(B, lane >> 4, i);  // axis 0 (lanes 0-15), axis 1 (lanes 16-31)
  const AxisScan C = scan_axis(B, 2, i);          // axis 2 (both halves)
  float best_cost[3];
  uint32_t best_count[3];
  best_cost[0] = __shfl_sync(0xffffffffu, A.best_cost, 0);
  best_count[0] = __shfl_sync(0xffffffffu, A.best_count, 0);
  best_cost[1] = __shfl_sync(0xffffffffu, A.best_cost, 16);
  best_count[1] = __shfl_sync(0xffffffffu, A.best_count, 16);
  best_cost[2] = C.best_cost;
  best_count[2] = C.best_count;
  int axis = 0;
  if (best_cost[0] > best_cost[1]) axis = 1;
  if (best_cost[axis] > best_cost[2]) axis = 2;
  uint32_t split_index = best_count[axis];
  const float max_split_cost = ha6(bmn, bmx) * ((float)ws - kTraversalCost);
  d.split = 0;
  if (best_count[axis] == (uint32_t)kBins || best_cost[axis] >= max_split_cost) {
    if (ws <= max_leaf) return;  // leaf
    // longest_axis (src/aabb.rs:353-363)
    int la = 0;
    if ((bmx[1] - bmn[1]) > (bmx[0] - bmn[0])) la = 1;
    if ((bmx[2] - bmn[2]) > (bmx[la] - bmn[la])) la = 2;
    axis = la;
    // first i < 15 whose cumulative count reaches ws * 2 / 5 + 1
    const uint64_t target = (uint64_t)ws * 2 / 5 + 1;
    const uint32_t mine = la == 2 ? C.pre.cnt : A.pre.cnt;
    const bool in_seg = la == 1 ? lane >= 16 : lane < 16;
    const uint32_t hit = __ballot_sync(0xffffffffu, in_seg && i < kBins - 1 && (uint64_t)mine >= target);
    if (hit) split_index = (uint32_t)(__ffs(hit) - 1 - (la == 1 ? 16 : 0)) + 1u;
  }
  const uint32_t n_left = fetch_cnt(A, C, axis, (int)min(split_index, (uint32_t)kBins) - 1);
  if (n_left == 0 || n_left >= ws) return;  // one side empty: leaf
  const int lb = (int)best_count[axis] - 1;     // bins [0, best_splits[axis].count)
  const int rb = (int)min(split_index, (uint32_t)kBins - 1u);  // bins [split_index, 16), split_index <= 15 here
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    d.lbox[f] = fetch_f(A, C, axis, lb, true, f);
    d.rbox[f] = fetch_f(A, C, axis, rb, false, f);
  }
  d.split = 1;
  d.axis = (uint32_t)axis;
  d.split_index = split_index;
  d.n_left = n_left;
}

__device__ __forceinline__ void init_bins(uint32_t* w, int tid, int nthreads) {
  const uint32_t kmin = float_to_ordered(1e34f), kmax = float_to_ordered(-1e34f);
  for (int i = tid; i < 3 * kBins; i += nthreads) {
    uint32_t* b = w + i * kBinWords;
    b[0] = b[1] = b[2] = kmin;
    b[3] = b[4] = b[5] = kmax;
    b[6] = 0;
    b[7] = 0;
  }
}

// Reads the node box, applies the first 1e-4 offset (binned_sah.rs:133),
// and writes it back (count/left_first untouched until the decision).
__device__ __forceinline__ void task_box(DAabb* nodes, uint32_t node, float mn[3], float mx[3]) {
  DAabb b = load_aabb_cg(nodes + node);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    mn[k] = b.min[k] - 0.0001f;
    mx[k] = b.max[k] + 0.0001f;
  }
}

// make_leaf (binned_sah.rs:134-138): second offset, left_first, count.
__device__ __forceinline__ void write_leaf(DAabb* nodes, const Task& t, const float mn[3], const float mx[3]) {
  DAabb b;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b.min[k] = mn[k] - 0.0001f;
    b.max[k] = mx[k] + 0.0001f;
  }
  b.count = (int32_t)(t.end - t.begin);
  b.left_first = (int32_t)t.begin;
  store_aabb(nodes + t.node, b);
}

__device__ __forceinline__ void write_interior_box(DAabb* nodes, uint32_t node, const float mn[3], const float mx[3]) {
  DAabb b;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b.min[k] = mn[k];
    b.max[k] = mx[k];
  }
  b.count = -1;
  b.left_first = -1;  // set by the emit kernel
  store_aabb(nodes + node, b);
}

struct SahParams {
  const DAabb* aabbs;
  const float4* centers;
  DAabb* nodes;
  uint32_t* idx_a;  // primitive indices (final output)
  uint32_t* idx_b;  // the other index array of the levels (see Level)
  uint32_t n;
  uint32_t max_leaf;
  uint32_t sub_max;     // largest task built as a subtree (<= kWarpMax)
  Task* large[2];       // task lists of even / odd levels
  Task* subs;           // subtree tasks (at most sub_max primitives), all levels
  void* tiny;           // SubTask list: subtrees of at most kSmall primitives (empty entries have end 0)
  uint32_t small_cap;   // its capacity
  void* mid;            // SubTask list: subtrees of at most kMid primitives (NULL: built in one go)
  uint32_t mid_cap;
  Decision* dec;        // large tasks of the level
  float* tbox;          // 6 floats per large task (box with first offset)
  uint32_t* bins;       // kTaskBinWords per large task
  uint32_t* chunk_base; // large + 1
  uint32_t* chunk_status;
  uint64_t* scan_vals;  // per task of the level
  uint64_t* scan_sums;  // one per block
  DAabb* tnodes;        // subtree node pairs by split position: 2(m-1), 2(m-1)+1
  uint32_t* sflag;      // 1 at the positions m where a subtree task splits
  uint32_t* srank;      // exclusive scan of sflag
  uint32_t* tile_off;   // per 4096-position tile: sums, then exclusive offsets
  Counters* cnt;
  GridBarrier* bar;
};

// The level being built, as every block read it after the level's first
// barrier.
struct Level {
  const Task* large;
  Task* large_next;
  uint32_t L, node_base, sub_base;
  uint32_t parity, next_parity;  // of this level and the next
  // Indices: a level reads its tasks' ranges from one array and leaves the
  // partitioned ranges in the other (idx_a at even levels, as the final
  // output is: a task that ends at an odd level is copied there).
  const uint32_t* src;
  uint32_t* dst;
};

// Reads of data written earlier in the same launch (by any block) go to L2:
// the L1 is not coherent between SMs.
__device__ __forceinline__ Task ld_task(const Task* t) {
  const uint4 v = __ldcg(reinterpret_cast<const uint4*>(t));
  return Task{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Decision ld_dec(const Decision* d) {
  Decision r;
  const uint4* q = reinterpret_cast<const uint4*>(d);
  uint4* o = reinterpret_cast<uint4*>(&r);
#pragma unroll
  for (int k = 0; k < 5; ++k) o[k] = __ldcg(q + k);
  return r;
}
__device__ __forceinline__ void ld_tbox(const float* tb, float mn[3], float mx[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = __ldcg(tb + a);
    mx[a] = __ldcg(tb + 3 + a);
  }
}

// Last t with chunk_base[t] <= chunk, 32 ways per read; all lanes of a warp
// call it.
__device__ __forceinline__ uint32_t find_task(const uint32_t* chunk_base, uint32_t L, uint32_t chunk) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lo = 0, n = L;  // the answer lies in [lo, lo + n)
  while (n > 1u) {
    const uint32_t step = (n + 31u) / 32u, at = lane * step;
    const uint32_t in = __ballot_sync(0xffffffffu, at < n && __ldcg(chunk_base + lo + at) <= chunk);
    const uint32_t k = (31u - __clz(in)) * step;  // lane 0 is always in
    lo += k;
    n = min(step, n - k);
  }
  return lo;
}

// Shared memory of one block, reused by the phases of a level. The fields
// are ordered by the phases that need them, so a launch of a single phase
// allocates only the prefix it uses (kShSmall, kShBins, all).
struct alignas(16) SahShared {
  uint64_t scan[kLargeBlock / 32];
  uint32_t warp[32];
  uint32_t chunk, fail, prefix, pad;
  uint32_t chunk_idx[kChunk];                      // the indices of a chunk
  uint32_t bins[kLargeBlock / 32][kTaskBinWords];  // per-warp bins
  Decision dec[kLargeBlock / 32];
  uint32_t idx[kLargeBlock / 32][kTaskWarp];       // per-warp partition buffer
};
constexpr size_t kShSmall = offsetof(SahShared, chunk_idx);  // scans, partition scalars
constexpr size_t kShChunk = offsetof(SahShared, bins);       // + a chunk's indices
constexpr size_t kShBins = offsetof(SahShared, dec);         // + a chunk's indices, per-warp bins

// Bins the primitives at positions [i0, i1) of every lane of a warp into `wb`
// (the warp's own shared bins; all 32 lanes call it). Neighbours in the index
// array are usually neighbours in space and share bins, so a lane merges a run
// of primitives in one bin in registers. At the end the lanes' last runs,
// which usually share a few bins, are merged over the warp bin by bin and
// written by one atomic per word; atomics of all lanes on one bin would take
// their turns. The next primitive is loaded before the current one is binned.
// What bounds it is the latency of these loads. One lane at a time and atomics
// of every lane took 58 us for an 800-primitive task of one warp.
template <class IdxFn>
__device__ __forceinline__ void bin_run(const SahParams& p, const BinMap& bm, uint32_t i0, uint32_t i1, IdxFn idx,
                                        uint32_t* wb) {
  constexpr uint32_t all = 0xffffffffu;
  uint32_t rbin[3], rmn[3][3], rmx[3][3], rcnt[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    rbin[a] = all;
    rcnt[a] = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      rmn[a][q] = all;
      rmx[a][q] = 0u;
    }
  }
  auto flush = [&](int a) {
    if (rcnt[a] == 0) return;
    uint32_t* b = wb + (a * kBins + rbin[a]) * kBinWords;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      atomicMin(b + q, rmn[a][q]);
      atomicMax(b + 3 + q, rmx[a][q]);
    }
    atomicAdd(b + 6, rcnt[a]);
  };
  float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  DAabb box = {};
  auto load = [&](uint32_t i) {
    const uint32_t prim = idx(i);
    c = __ldg(p.centers + prim);
    box = load_aabb(p.aabbs + prim);
  };
  if (i0 < i1) load(i0);
#pragma unroll 1
  for (uint32_t i = i0; i < i1; ++i) {
    const float cc[3] = {c.x, c.y, c.z};
    uint32_t kmn[3], kmx[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      kmn[q] = float_to_ordered(box.min[q]);
      kmx[q] = float_to_ordered(box.max[q]);
    }
    if (i + 1u < i1) load(i + 1u);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t bin = bin_of(cc[a], bm.c2b[a], bm.off[a]);
      if (bin != rbin[a]) {
        flush(a);
        rbin[a] = bin;
        rcnt[a] = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          rmn[a][q] = kmn[q];
          rmx[a][q] = kmx[q];
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        rmn[a][q] = min(rmn[a][q], kmn[q]);
        rmx[a][q] = max(rmx[a][q], kmx[q]);
      }
      ++rcnt[a];
    }
  }
  __syncwarp();
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    uint32_t pending = __ballot_sync(all, rcnt[a] != 0u);
    // bins that four lanes or more hold, as long as many lanes are left
#pragma unroll 1
    for (int round = 0; round < 4 && __popc(pending) >= 8; ++round) {
      const uint32_t b = __shfl_sync(all, rbin[a], __ffs(pending) - 1);
      const bool in = rcnt[a] != 0u && rbin[a] == b;
      const uint32_t group = __ballot_sync(all, in);
      if (__popc(group) < 4) break;
      uint32_t v = 0;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t mn = __reduce_min_sync(all, in ? rmn[a][q] : all);
        const uint32_t mx = __reduce_max_sync(all, in ? rmx[a][q] : 0u);
        if (lane == (uint32_t)q) v = mn;
        if (lane == 3u + (uint32_t)q) v = mx;
      }
      const uint32_t n = __reduce_add_sync(all, in ? rcnt[a] : 0u);
      uint32_t* w = wb + (a * kBins + b) * kBinWords + lane;
      if (lane < 3u) atomicMin(w, v);
      else if (lane < 6u) atomicMax(w, v);
      else if (lane == 6u) atomicAdd(w, n);
      if (in) rcnt[a] = 0u;
      pending &= ~group;
    }
    flush(a);
  }
}

// ------------------------------------------------------------------ large tasks
// Block 0: task boxes (with the first 1e-4 offset) and chunk offsets of the
// level's large tasks.
// `above`: tasks of at most so many primitives get no chunks (a warp does them).
__device__ void large_prep(const SahParams& p, const Level& lv, SahShared& sh, uint32_t above) {
  uint32_t carry = 0;
  for (uint32_t base = 0; base < lv.L; base += kLargeBlock) {
    const uint32_t t = base + threadIdx.x;
    uint32_t chunks = 0;
    if (t < lv.L) {
      const Task tk = ld_task(lv.large + t);
      float mn[3], mx[3];
      task_box(p.nodes, tk.node, mn, mx);
      float* tb = p.tbox + 6 * (size_t)t;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        tb[k] = mn[k];
        tb[3 + k] = mx[k];
      }
      const uint32_t ws = tk.end - tk.begin;
      if (ws > above && tk.depth < kMaxDepth) chunks = (ws + kChunk - 1) / kChunk;
    }
    uint32_t total;
    const uint32_t incl = block_inclusive_scan<kLargeBlock>(chunks, sh.warp, &total);
    if (t < lv.L) p.chunk_base[t] = carry + incl - chunks;
    carry += total;
  }
  if (threadIdx.x == 0) {
    p.chunk_base[lv.L] = carry;
    p.cnt->chunks = carry;
    p.cnt->ticket = 0;
  }
}

// Empty bins for every large task (one bin per thread of the grid).
__device__ void large_bins_init(const SahParams& p, const Level& lv) {
  const uint32_t kmin = float_to_ordered(1e34f), kmax = float_to_ordered(-1e34f);
  const size_t total = (size_t)lv.L * 3 * kBins;
  for (size_t i = (size_t)blockIdx.x * kLargeBlock + threadIdx.x; i < total; i += (size_t)gridDim.x * kLargeBlock) {
    uint4* b = reinterpret_cast<uint4*>(p.bins + i * kBinWords);
    b[0] = make_uint4(kmin, kmin, kmin, kmax);
    b[1] = make_uint4(kmax, kmax, 0u, 0u);
  }
}

// Bins one 2048-primitive chunk of a large task into the task's global bins.
__device__ void large_bin_chunk(const SahParams& p, const Level& lv, uint32_t chunk, SahShared& sh) {
  const int warp = threadIdx.x >> 5;
  const uint32_t t = find_task(p.chunk_base, lv.L, chunk);
  const Task tk = ld_task(lv.large + t);
  const uint32_t k = chunk - __ldcg(p.chunk_base + t);
  const uint32_t c0 = tk.begin + k * kChunk;
  const uint32_t c1 = min(c0 + kChunk, tk.end);
  init_bins(&sh.bins[warp][0], threadIdx.x & 31, 32);
  for (uint32_t i = c0 + threadIdx.x; i < c1; i += kLargeBlock) sh.chunk_idx[i - c0] = __ldcg(lv.src + i);
  __syncthreads();
  float mn[3], mx[3];
  ld_tbox(p.tbox + 6 * (size_t)t, mn, mx);
  const BinMap bm = make_binmap(mn, mx);
  uint32_t* wb = &sh.bins[warp][0];
  // each thread bins kChunk / kLargeBlock consecutive primitives
  constexpr uint32_t PER = kChunk / kLargeBlock;
  const uint32_t s0 = c0 + threadIdx.x * PER;
  bin_run(p, bm, min(s0, c1), min(s0 + PER, c1), [&](uint32_t i) { return sh.chunk_idx[i - c0]; }, wb);
  __syncthreads();
  uint32_t* gb = p.bins + (size_t)t * kTaskBinWords;
  for (int i = threadIdx.x; i < 3 * kBins; i += kLargeBlock) {
    uint32_t cnt = 0;
    uint32_t vmn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, vmx[3] = {0u, 0u, 0u};
    for (int w = 0; w < kLargeBlock / 32; ++w) {
      const uint32_t* b = &sh.bins[w][i * kBinWords];
      cnt += b[6];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        vmn[q] = min(vmn[q], b[q]);
        vmx[q] = max(vmx[q], b[3 + q]);
      }
    }
    if (cnt) {
      uint32_t* g = gb + i * kBinWords;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        atomicMin(g + q, vmn[q]);
        atomicMax(g + 3 + q, vmx[q]);
      }
      atomicAdd(g + 6, cnt);
    }
  }
  __syncthreads();  // the shared bins are reused by the block's next chunk
}

// Split decision of large task t by one warp (its global bins are copied to
// the warp's shared bins first).
__device__ void large_decide(const SahParams& p, const Level& lv, uint32_t t, SahShared& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Task tk = ld_task(lv.large + t);
  float mn[3], mx[3];
  ld_tbox(p.tbox + 6 * (size_t)t, mn, mx);
  Decision d;
  d.split = 0;
  const uint32_t ws = tk.end - tk.begin;
  if (ws > 1 && tk.depth < kMaxDepth) {
    uint32_t* wb = &sh.bins[warp][0];
    const uint32_t* gb = p.bins + (size_t)t * kTaskBinWords;
    for (int i = lane; i < kTaskBinWords; i += 32) wb[i] = __ldcg(gb + i);
    __syncwarp();
    sah_decide_warp(BinsView{wb}, mn, mx, ws, p.max_leaf, d);
    __syncwarp();
  }
  if (lane == 0) {
    if (d.split) write_interior_box(p.nodes, tk.node, mn, mx);
    else write_leaf(p.nodes, tk, mn, mx);
    p.dec[t] = d;
  }
}

// Task t whole -- bins, decision and partition -- by one warp (at most kTaskWarp
// primitives) or by the block (at most a chunk).
__device__ void large_task_warp(const SahParams& p, const Level& lv, uint32_t t, SahShared& sh);
__device__ void large_task_block(const SahParams& p, const Level& lv, uint32_t t, SahShared& sh);

// Stable partition of a large task's chunk from lv.src to lv.dst; the number of
// left primitives in the task's earlier chunks comes from a decoupled look-back,
// 32 chunks at a time
// (chunks are taken in ticket order, so every chunk waited on is held by a
// running block).
__device__ void large_partition_chunk(const SahParams& p, const Level& lv, uint32_t chunk, SahShared& sh) {
  const uint32_t t = find_task(p.chunk_base, lv.L, chunk);
  const Decision d = ld_dec(p.dec + t);
  const Task tk = ld_task(lv.large + t);
  const uint32_t first_chunk = __ldcg(p.chunk_base + t);
  const uint32_t k = chunk - first_chunk;
  const uint32_t c0 = tk.begin + k * kChunk;
  const uint32_t c1 = min(c0 + kChunk, tk.end);
  if (!d.split) {  // no chunk of this task waits on another
    if (lv.parity)
      for (uint32_t i = c0 + threadIdx.x; i < c1; i += kLargeBlock) p.idx_a[i] = __ldcg(lv.src + i);
    return;
  }
  for (uint32_t i = c0 + threadIdx.x; i < c1; i += kLargeBlock) sh.chunk_idx[i - c0] = __ldcg(lv.src + i);
  float mn[3], mx[3];
  ld_tbox(p.tbox + 6 * (size_t)t, mn, mx);
  const BinMap bm = make_binmap(mn, mx);
  const int ax = (int)d.axis;
  constexpr int PER = kChunk / kLargeBlock;
  uint32_t prim[PER];
  uint32_t flags = 0, mine = 0;
  const uint32_t s = c0 + threadIdx.x * PER;
  __syncthreads();
  float cc[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const uint32_t i = s + j;
    prim[j] = 0;
    cc[j] = 0.0f;
    if (i < c1) {
      prim[j] = sh.chunk_idx[i - c0];
      cc[j] = __ldg(reinterpret_cast<const float*>(p.centers + prim[j]) + ax);
    }
  }
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    if (s + j < c1 && bin_of(cc[j], bm.c2b[ax], bm.off[ax]) < d.split_index) {
      flags |= 1u << j;
      ++mine;
    }
  }
  uint32_t chunk_true;
  const uint32_t incl = block_inclusive_scan<kLargeBlock>(mine, sh.warp, &chunk_true);
  const uint32_t before_me = incl - mine;
  volatile uint32_t* st = p.chunk_status;
  if (threadIdx.x < 32) {  // 32 earlier chunks per look
    const uint32_t lane = threadIdx.x;
    uint32_t excl = 0;
    bool ok = true;
    if (lane == 0) st[chunk] = (k == 0 ? kFlagInc : kFlagAgg) | chunk_true;
    for (uint32_t end = chunk; end > first_chunk && ok;) {  // chunks [first_chunk, end) are to be added
      const bool there = end - first_chunk > lane;
      uint32_t v = 0, spins = 0;
      if (there) {
        while (((v = st[end - 1u - lane]) & ~kCountMask) == 0u) {
          if (++spins > kSpinLimit) break;
          __nanosleep(32);
        }
      }
      ok = __all_sync(0xffffffffu, !there || (v & ~kCountMask) != 0u);
      const uint32_t incs = __ballot_sync(0xffffffffu, there && (v & ~kCountMask) == kFlagInc);
      const uint32_t last = incs ? (uint32_t)__ffs(incs) - 1u : 31u;  // the nearest inclusive count
      excl += __reduce_add_sync(0xffffffffu, there && lane <= last ? v & kCountMask : 0u);
      if (incs) break;
      end -= min(32u, end - first_chunk);
    }
    if (lane == 0) {
      if (!ok) atomicOr(&p.cnt->status, kStatusTimeout);
      else if (k > 0) st[chunk] = kFlagInc | (excl + chunk_true);
      sh.fail = ok ? 0u : 1u;
      sh.prefix = excl;
    }
  }
  __syncthreads();
  const bool fail = sh.fail != 0;
  const uint32_t true_before = sh.prefix;
  // the chunk's left ones to the front of the staged indices, in order
  uint32_t tl = before_me, fl = chunk_true + (threadIdx.x * PER - before_me);
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (s + j < c1) sh.chunk_idx[((flags >> j) & 1u) ? tl++ : fl++] = prim[j];
  __syncthreads();
  if (fail) return;
  const uint32_t left_at = tk.begin + true_before;
  const uint32_t right_at = tk.begin + d.n_left + ((c0 - tk.begin) - true_before);
  for (uint32_t i = threadIdx.x; i < c1 - c0; i += kLargeBlock) {
    const uint32_t dst = i < chunk_true ? left_at + i : right_at + (i - chunk_true);
    if (dst < tk.end) lv.dst[dst] = sh.chunk_idx[i];
    else atomicOr(&p.cnt->status, kStatusBadIndex);
  }
  __syncthreads();  // the staged indices are rewritten by the block's next chunk
}

// ------------------------------------------------------------------ small tasks
// Subtrees of at most kSmall primitives are listed and built by k_sub_small.
// 4M clustered triangles, build with both trees: 8 primitives 9.44 ms, 12
// 9.20, 16 9.20, 24 9.58, 32 9.86.
constexpr uint32_t kSmall = 16;
static_assert(kSmall <= 32, "a lane per primitive");

// BinnedSahBuildTask::run (binned_sah.rs:132-282) after the node box is known,
// for a task of more than kSmall primitives by one warp: bins in shared memory
// (wb), indices staged in sidx, the warp-parallel decision, a ballot-based
// stable partition. The decision is left in `d` (shared
// memory, written by lane 0) for every lane.
// The indices are read from src and written, partitioned, to dst (which may be
// the same).
__device__ void decide_warp(const SahParams& p, const uint32_t* src, uint32_t* dst_idx, uint32_t begin, uint32_t ws,
                            uint32_t depth, const float mn[3], const float mx[3], uint32_t* wb, uint32_t* sidx,
                            Decision& d) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) d.split = 0;
  __syncwarp();
  if (ws > 1 && depth < kMaxDepth && ws <= kWarpMax) {
    init_bins(wb, lane, 32);
    // stage the task's indices (independent loads, all in flight at once)
    for (uint32_t i = lane; i < ws; i += 32) sidx[i] = __ldcg(src + begin + i);
    __syncwarp();
    const BinMap bm = make_binmap(mn, mx);
    {
      // each lane bins a contiguous slice, merging runs of primitives that
      // fall in one bin before its shared-memory atomics
      const uint32_t per = (ws + 31) / 32;
      const uint32_t lo = min(ws, (uint32_t)lane * per);
      bin_run(p, bm, lo, min(ws, lo + per), [&](uint32_t i) { return sidx[i]; }, wb);
    }
    __syncwarp();
    {
      Decision dl;
      sah_decide_warp(BinsView{wb}, mn, mx, ws, p.max_leaf, dl);
      if (lane == 0) d = dl;
    }
    __syncwarp();
    if (d.split) {
      const int ax = (int)d.axis;
      const uint32_t lt = (1u << lane) - 1u;
      const uint32_t split_index = d.split_index, n_left = d.n_left;
      uint32_t tb = 0, fb = 0;
      for (uint32_t c0 = 0; c0 < ws; c0 += 32) {
        const uint32_t i = c0 + lane;
        const bool valid = i < ws;
        uint32_t prim = 0;
        bool pred = false;
        if (valid) {
          prim = sidx[i];
          const float4 c = __ldg(p.centers + prim);
          const float cc = ax == 0 ? c.x : (ax == 1 ? c.y : c.z);
          pred = bin_of(cc, bm.c2b[ax], bm.off[ax]) < split_index;
        }
        const uint32_t T = __ballot_sync(0xffffffffu, pred);
        const uint32_t V = __ballot_sync(0xffffffffu, valid);
        const uint32_t F = V & ~T;
        // written straight to the task's range: the staged copy is the source
        if (pred) dst_idx[begin + tb + __popc(T & lt)] = prim;
        else if (valid) {
          const uint32_t dst = n_left + fb + __popc(F & lt);
          if (dst < ws) dst_idx[begin + dst] = prim;
        }
        tb += __popc(T);
        fb += __popc(F);
      }
    }
  }
  __syncwarp();
}

__device__ void large_task_warp(const SahParams& p, const Level& lv, uint32_t t, SahShared& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Task tk = ld_task(lv.large + t);
  float mn[3], mx[3];
  task_box(p.nodes, tk.node, mn, mx);
  decide_warp(p, lv.src, lv.dst, tk.begin, tk.end - tk.begin, tk.depth, mn, mx, sh.bins[warp], sh.idx[warp],
              sh.dec[warp]);
  if (lv.parity && !sh.dec[warp].split)  // (a task at the depth limit ends at an even level)
    for (uint32_t i = tk.begin + lane; i < tk.end; i += 32) p.idx_a[i] = __ldcg(lv.src + i);
  if (lane == 0) {
    if (sh.dec[warp].split) write_interior_box(p.nodes, tk.node, mn, mx);
    else write_leaf(p.nodes, tk, mn, mx);
    p.dec[t] = sh.dec[warp];
  }
  __syncwarp();
}

__device__ void large_task_block(const SahParams& p, const Level& lv, uint32_t t, SahShared& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Task tk = ld_task(lv.large + t);
  const uint32_t ws = tk.end - tk.begin;
  float mn[3], mx[3];
  task_box(p.nodes, tk.node, mn, mx);
  if (threadIdx.x == 0) sh.dec[0].split = 0;
  if (ws > 1 && tk.depth < kMaxDepth) {
    init_bins(&sh.bins[warp][0], lane, 32);
    for (uint32_t i = threadIdx.x; i < ws; i += kLargeBlock) sh.chunk_idx[i] = __ldcg(lv.src + tk.begin + i);
    __syncthreads();
    const BinMap bm = make_binmap(mn, mx);
    const uint32_t per = (ws + kLargeBlock - 1) / kLargeBlock;
    const uint32_t i0 = min(threadIdx.x * per, ws), i1 = min(i0 + per, ws);
    bin_run(p, bm, i0, i1, [&](uint32_t i) { return sh.chunk_idx[i]; }, &sh.bins[warp][0]);
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * kBins; i += kLargeBlock) {
      uint32_t* b0 = &sh.bins[0][i * kBinWords];
      for (int w = 1; w < kLargeBlock / 32; ++w) {
        const uint32_t* b = &sh.bins[w][i * kBinWords];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          b0[q] = min(b0[q], b[q]);
          b0[3 + q] = max(b0[3 + q], b[3 + q]);
        }
        b0[6] += b[6];
      }
    }
    __syncthreads();
    if (warp == 0) {
      Decision d;
      sah_decide_warp(BinsView{&sh.bins[0][0]}, mn, mx, ws, p.max_leaf, d);
      if (lane == 0) sh.dec[0] = d;
    }
    __syncthreads();
    if (sh.dec[0].split) {
      const int ax = (int)sh.dec[0].axis;
      const uint32_t split_index = sh.dec[0].split_index;
      uint32_t flags = 0, mine = 0;  // per <= 8
      for (uint32_t i = i0; i < i1; ++i) {
        const float4 c = __ldg(p.centers + sh.chunk_idx[i]);
        const float cc = ax == 0 ? c.x : (ax == 1 ? c.y : c.z);
        if (bin_of(cc, bm.c2b[ax], bm.off[ax]) < split_index) {
          flags |= 1u << (i - i0);
          ++mine;
        }
      }
      uint32_t total;
      const uint32_t before = block_inclusive_scan<kLargeBlock>(mine, sh.warp, &total) - mine;
      uint32_t tpos = tk.begin + before, fpos = tk.begin + sh.dec[0].n_left + (i0 - before);
      for (uint32_t i = i0; i < i1; ++i) {
        const uint32_t dst = ((flags >> (i - i0)) & 1u) ? tpos++ : fpos++;
        if (dst < tk.end) lv.dst[dst] = sh.chunk_idx[i];
        else atomicOr(&p.cnt->status, kStatusBadIndex);
      }
    } else if (lv.parity) {
      for (uint32_t i = threadIdx.x; i < ws; i += kLargeBlock) p.idx_a[tk.begin + i] = sh.chunk_idx[i];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (sh.dec[0].split) write_interior_box(p.nodes, tk.node, mn, mx);
    else write_leaf(p.nodes, tk, mn, mx);
    p.dec[t] = sh.dec[0];
  }
  __syncthreads();
}

// ------------------------------------------------------------------ subtrees
constexpr uint32_t kTemp = 0x80000000u;  // SubTask::loc bit: a scratch slot, else a node of the breadth-first part

struct SubTask {
  uint32_t loc, begin, end, depth;
  float box[6];  // the box the parent gave the node (min xyz, max xyz), before the first offset
};
constexpr int kSubStack = (int)kMaxDepth + 2;
constexpr int kSubBlock = 128;

// Shared memory of one warp of k_sub_build.
struct SubShared {
  uint32_t bins[kTaskBinWords];
  uint32_t idx[kWarpMax];
  Decision dec;
  SubTask stack[kSubStack];
};

__device__ __forceinline__ DAabb* sub_node(const SahParams& p, uint32_t loc) {
  return (loc & kTemp) ? p.tnodes + (loc & ~kTemp) : p.nodes + loc;
}

// Writes task tk's node (mn / mx: its box with the first offset): an
// interior node whose left_first is, until the relocation, the split
// position m; or a leaf (make_leaf: second offset, first primitive, count).
// On a split, notes m and returns the children.
__device__ __forceinline__ bool sub_write(const SahParams& p, const SubTask& tk, const float mn[3], const float mx[3],
                                          const Decision& d, SubTask& l, SubTask& r) {
  DAabb b;
  if (d.split) {
    const uint32_t m = tk.begin + d.n_left;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      b.min[k] = mn[k];
      b.max[k] = mx[k];
    }
    b.count = -1;
    b.left_first = (int32_t)m;
    store_aabb(sub_node(p, tk.loc), b);
    p.sflag[m] = 1u;
    l.loc = kTemp | (2u * (m - 1u));
    l.begin = tk.begin;
    l.end = m;
    l.depth = tk.depth + 1u;
    r.loc = kTemp | (2u * (m - 1u) + 1u);
    r.begin = m;
    r.end = tk.end;
    r.depth = tk.depth + 1u;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      l.box[k] = d.lbox[k];
      r.box[k] = d.rbox[k];
    }
    return true;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    b.min[k] = mn[k] - 0.0001f;
    b.max[k] = mx[k] + 0.0001f;
  }
  b.count = (int32_t)(tk.end - tk.begin);
  b.left_first = (int32_t)tk.begin;
  store_aabb(sub_node(p, tk.loc), b);
  return false;
}

__device__ __forceinline__ void first_offset(const SubTask& tk, float mn[3], float mx[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    mn[k] = tk.box[k] - 0.0001f;
    mx[k] = tk.box[3 + k] + 0.0001f;
  }
}

// A list of subtrees that warps append to, each reserving CHUNK entries at a
// time: one atomic per so many subtrees. What is left over when the warp ends
// is marked empty.
template <uint32_t CHUNK>
struct SubList {
  SubTask* entries;
  uint32_t cap;
  uint32_t* count;
  uint32_t next = 0, end = 0;
  __device__ __forceinline__ SubList(void* list, uint32_t capacity, uint32_t* counter)
      : entries(reinterpret_cast<SubTask*>(list)), cap(capacity), count(counter) {}
  // by one lane of the warp
  __device__ __forceinline__ void add(const SahParams& p, const SubTask& t) {
    if (next == end) {
      next = atomicAdd(count, CHUNK);
      end = next + CHUNK;
    }
    if (next < cap) entries[next] = t;
    else atomicOr(&p.cnt->status, kStatusBadIndex);
    ++next;
  }
  __device__ __forceinline__ void finish() {
    for (; next < end && next < cap; ++next) {
      SubTask t = {};
      entries[next] = t;
    }
  }
};
constexpr uint32_t kListChunk = 32, kMidChunk = 4;
using SmallList = SubList<kListChunk>;
using MidList = SubList<kMidChunk>;

// Builds with subtrees of more than kMidFrom primitives build them in two
// launches: the first splits every subtree until its parts are at most kMid,
// the second builds the parts. In one, a warp that has a whole subtree of up
// to 1,024 primitives is busy for a third of the launch, and there are fewer
// than three of them for each. 4M clustered triangles in one launch 8,077 us;
// kMid 512: 8,047, 256: 7,871, 128: 7,828, 64: 7,871; 700k 2,345 in one, 2,285
// in two, 520k 2,028 and 1,960, 400k 1,824 and 1,772, but 300k 1,504 and 1,500,
// 270k 1,452 and 1,471. Five or six blocks per SM (102 or 80 registers) and
// less shared memory in the second launch: no faster.
constexpr uint32_t kMid = 128, kMidFrom = 160;

// One subtree (index array of its level in idx_a) by one warp, depth first:
// tasks of more than kSmall primitives by the whole warp; smaller ones are
// listed for k_sub_small and, with SPLIT, those of up to kMid for the second
// launch. Every write goes to a place fixed by the task's primitive range, so
// the order in which tasks run does not matter.
template <bool SPLIT>
__device__ void sub_warp_tree(const SahParams& p, const SubTask& root, SubShared& sh, SmallList& list, MidList& mids) {
  const int lane = threadIdx.x & 31;
  int sp = -1;  // warp-uniform
  // true where the task goes onto the stack; by all lanes, with the same task
  auto keep = [&](uint32_t size, const SubTask& t) {
    if (size <= kSmall) {
      if (lane == 0) list.add(p, t);
    } else if (SPLIT && size <= kMid) {
      if (lane == 0) mids.add(p, t);
    } else {
      if (lane == 0) sh.stack[sp + 1] = t;
      return true;
    }
    return false;
  };
  if (keep(root.end - root.begin, root)) sp = 0;
  __syncwarp();
  while (sp >= 0) {
    const SubTask tk = sh.stack[sp--];
    float mn[3], mx[3];
    first_offset(tk, mn, mx);
    decide_warp(p, p.idx_a, p.idx_a, tk.begin, tk.end - tk.begin, tk.depth, mn, mx, sh.bins, sh.idx, sh.dec);
    const Decision d = sh.dec;
    __syncwarp();
    SubTask l, r;
    if (lane == 0) sub_write(p, tk, mn, mx, d, l, r);
    if (d.split) {
      const uint32_t nl = d.n_left, nr = (tk.end - tk.begin) - d.n_left;
      if (sp + 2 >= kSubStack) {
        if (lane == 0) atomicOr(&p.cnt->status, kStatusBadIndex);
        return;
      }
      // right child first onto the stack: the left one is taken next
      if (keep(nr, r)) ++sp;
      if (keep(nl, l)) ++sp;
    }
    __syncwarp();
  }
}

// The listed subtree t of the breadth-first part, with its indices in idx_a.
__device__ __forceinline__ SubTask sub_root(const SahParams& p, const Task& root) {
  // a subtree that hangs below an even level has its indices in idx_b
  if (root.depth & 1u)
    for (uint32_t i = root.begin + (threadIdx.x & 31u); i < root.end; i += 32) p.idx_a[i] = __ldcg(p.idx_b + i);
  __syncwarp();
  const DAabb rb = load_aabb_cg(p.nodes + root.node);
  SubTask t;
  t.loc = root.node;
  t.begin = root.begin;
  t.end = root.end;
  t.depth = root.depth;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    t.box[k] = rb.min[k];
    t.box[3 + k] = rb.max[k];
  }
  return t;
}

// ------------------------------------------------------------------ subtrees of at most kSmall primitives
// Shared memory of one warp of k_sub_small: the primitives in lane order, their
// boxes ({min, bins}, {max, primitive}; w as integers) and centres.
struct SmallShared {
  float4 lo[32], hi[32];
  float4 centre[32];
  uint8_t entry[32];  // list entry that starts at a lane
};

// (cost key, bin) pairs: the smaller first.
__device__ __forceinline__ bool pair_less(uint32_t a, uint32_t ab, uint32_t b, uint32_t bb) {
  return a < b || (a == b && ab < bb);
}

// Several subtrees at once, one primitive per lane: a task is a run of lanes
// [s, e), its children are the runs its stable partition leaves, so all tasks
// of a level are decided side by side (BinnedSahBuildTask::run,
// binned_sah.rs:132-282). There are no bins: find_split's cost at bin i
// depends only on which primitives lie left and right of i -- it is NaN while
// a side is empty and constant between two non-empty bins -- so every lane
// evaluates the cost at its own primitive's bin of each axis, over the boxes of
// its run (the same unions, hence the same bits), and the first minimum is the
// smallest (cost, bin) pair of the run. What bounds it is instruction issue
// (60 % of the slots), about 50 per member of the longest run and 500 per
// level. Before, subtrees of at most 8 primitives took a thread each, which
// left 114 us of latency at 6,400 triangles (34 now).
__device__ void small_subtrees(const SahParams& p, SmallShared& sh, bool valid, SubTask tk, uint32_t first_lane) {
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t all = 0xffffffffu;
  uint32_t s = first_lane, e = first_lane + (tk.end - tk.begin);
  const uint32_t pos = tk.begin + (lane - first_lane);  // the lane's index slot
  if (valid) {
    const uint32_t prim = p.idx_a[pos];
    const DAabb b = load_aabb(p.aabbs + prim);
    sh.centre[lane] = __ldg(p.centers + prim);
    sh.lo[lane] = make_float4(b.min[0], b.min[1], b.min[2], 0.0f);
    sh.hi[lane] = make_float4(b.max[0], b.max[1], b.max[2], __uint_as_float(prim));
  }
  bool open = valid;  // the lane's task is not finished
  while (__any_sync(all, open)) {
    const uint32_t ws = open ? e - s : 0u;
    float mn[3], mx[3];
    first_offset(tk, mn, mx);
    const bool decide = open && ws > 1u && tk.depth < kMaxDepth;
    uint32_t packed = 0;
    __syncwarp();
    if (decide) {
      const BinMap bm = make_binmap(mn, mx);
      const float4 c = sh.centre[lane];
      packed = bin_of(c.x, bm.c2b[0], bm.off[0]) | bin_of(c.y, bm.c2b[1], bm.off[1]) << 4 |
               bin_of(c.z, bm.c2b[2], bm.off[2]) << 8;
      sh.lo[lane].w = __uint_as_float(packed);
    }
    __syncwarp();
    // costs at the own primitive's bins (areas: the sign of a zero does not
    // matter, native min/max will do)
    float lmn[3][3], lmx[3][3], rmn[3][3], rmx[3][3];
    uint32_t nl[3] = {0u, 0u, 0u};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lmn[a][k] = rmn[a][k] = 1e34f;
        lmx[a][k] = rmx[a][k] = -1e34f;
      }
    const uint32_t members = decide ? ws : 0u;
    const uint32_t longest = __reduce_max_sync(all, members);
    for (uint32_t k = 0; k < members; ++k) {
      const float4 lo = sh.lo[s + k], hi = sh.hi[s + k];
      const uint32_t bins = __float_as_uint(lo.w);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const bool left = (bins >> (4 * a) & 15u) <= (packed >> (4 * a) & 15u);
        if (left) {
          ++nl[a];
          lmn[a][0] = fminf(lmn[a][0], lo.x); lmn[a][1] = fminf(lmn[a][1], lo.y); lmn[a][2] = fminf(lmn[a][2], lo.z);
          lmx[a][0] = fmaxf(lmx[a][0], hi.x); lmx[a][1] = fmaxf(lmx[a][1], hi.y); lmx[a][2] = fmaxf(lmx[a][2], hi.z);
        } else {
          rmn[a][0] = fminf(rmn[a][0], lo.x); rmn[a][1] = fminf(rmn[a][1], lo.y); rmn[a][2] = fminf(rmn[a][2], lo.z);
          rmx[a][0] = fmaxf(rmx[a][0], hi.x); rmx[a][1] = fmaxf(rmx[a][1], hi.y); rmx[a][2] = fmaxf(rmx[a][2], hi.z);
        }
      }
    }
    __syncwarp();
    float best_cost[3];
    uint32_t best_count[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      uint32_t key = all, bin = (uint32_t)kBins;  // none: above every cost below f32::MAX
      if (decide && nl[a] < ws) {
        const float cost = ha6(lmn[a], lmx[a]) * (float)nl[a] + ha6(rmn[a], rmx[a]) * (float)(ws - nl[a]);
        if (cost < kF32Max) {
          key = float_to_ordered(cost + 0.0f);  // -0 and +0 compare equal
          bin = packed >> (4 * a) & 15u;
        }
      }
      // smallest pair of the run: inclusive over [s, lane], then the last lane's
#pragma unroll 1
      for (uint32_t o = 1; o < longest; o <<= 1) {
        const uint32_t ok = __shfl_up_sync(all, key, o), ob = __shfl_up_sync(all, bin, o);
        if (lane >= s + o && pair_less(ok, ob, key, bin)) {
          key = ok;
          bin = ob;
        }
      }
      const uint32_t last = (e - 1u) & 31u;
      key = __shfl_sync(all, key, last);
      bin = __shfl_sync(all, bin, last);
      best_cost[a] = bin < (uint32_t)kBins ? ordered_to_float(key) : kF32Max;
      best_count[a] = bin < (uint32_t)kBins ? bin + 1u : (uint32_t)kBins;
    }
    int axis = 0;
    if (best_cost[0] > best_cost[1]) axis = 1;
    if ((axis ? best_cost[1] : best_cost[0]) > best_cost[2]) axis = 2;
    uint32_t split_index = axis == 0 ? best_count[0] : (axis == 1 ? best_count[1] : best_count[2]);
    const float cost = axis == 0 ? best_cost[0] : (axis == 1 ? best_cost[1] : best_cost[2]);
    const float max_split_cost = ha6(mn, mx) * ((float)ws - kTraversalCost);
    const bool fallback = decide && (split_index == (uint32_t)kBins || cost >= max_split_cost);
    bool leaf = !decide;
    if (__any_sync(all, fallback)) {
      int la = 0;
      if ((mx[1] - mn[1]) > (mx[0] - mn[0])) la = 1;
      if ((mx[2] - mn[2]) > (la ? mx[1] - mn[1] : mx[0] - mn[0])) la = 2;
      // the first bin below 15 whose cumulative count reaches ws * 2 / 5 + 1
      const uint32_t bin = packed >> (4 * la) & 15u, upto = la == 0 ? nl[0] : (la == 1 ? nl[1] : nl[2]);
      uint32_t b = fallback && bin < (uint32_t)kBins - 1u && upto >= ws * 2u / 5u + 1u ? bin : (uint32_t)kBins;
#pragma unroll 1
      for (uint32_t o = 1; o < longest; o <<= 1) {
        const uint32_t ob = __shfl_up_sync(all, b, o);
        if (lane >= s + o) b = min(b, ob);
      }
      b = __shfl_sync(all, b, (e - 1u) & 31u);
      if (fallback) {
        if (ws <= p.max_leaf) {
          leaf = true;
        } else {
          axis = la;
          if (b < (uint32_t)kBins) split_index = b + 1u;
        }
      }
    }
    const uint32_t mine = packed >> (4 * axis) & 15u;
    const bool goes_left = decide && !leaf && mine < split_index;
    const uint32_t run = open ? (all >> (32u - ws)) << s : 0u;
    const uint32_t lefts = __ballot_sync(all, goes_left) & run;
    const uint32_t n_left = __popc(lefts);
    const bool split = open && !leaf && n_left > 0u && n_left < ws;
    // the children's boxes: left over the bins below best_count of the axis (a
    // quirk of the reference), right over the bins from split_index
    const uint32_t lcount = axis == 0 ? best_count[0] : (axis == 1 ? best_count[1] : best_count[2]);
    uint32_t cmn[3], cmx[3];  // ordered keys: the boxes' bits count here
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      cmn[k] = float_to_ordered(1e34f);
      cmx[k] = float_to_ordered(-1e34f);
    }
    const uint32_t more = split ? ws : 0u;
    for (uint32_t k = 0; k < more; ++k) {
      const float4 lo = sh.lo[s + k], hi = sh.hi[s + k];
      const uint32_t b = __float_as_uint(lo.w) >> (4 * axis) & 15u;
      if (goes_left ? b < lcount : b >= split_index) {
        cmn[0] = min(cmn[0], float_to_ordered(lo.x));
        cmn[1] = min(cmn[1], float_to_ordered(lo.y));
        cmn[2] = min(cmn[2], float_to_ordered(lo.z));
        cmx[0] = max(cmx[0], float_to_ordered(hi.x));
        cmx[1] = max(cmx[1], float_to_ordered(hi.y));
        cmx[2] = max(cmx[2], float_to_ordered(hi.z));
      }
    }
    __syncwarp();
    if (open && lane == s) {
      Decision d;
      d.split = split ? 1u : 0u;
      d.n_left = n_left;
      SubTask l, r;
      sub_write(p, tk, mn, mx, d, l, r);
    }
    uint32_t to = lane;
    if (split) {
      const uint32_t before = (1u << lane) - 1u;
      to = goes_left ? s + __popc(lefts & before) : s + n_left + __popc(run & ~lefts & before);
    }
    // the lane's new primitive and task (its own where nothing moved)
    const float4 lo = sh.lo[lane], hi = sh.hi[lane], c = sh.centre[lane];
    // both children's boxes, from a lane of either side
    const uint32_t lsrc = split ? (uint32_t)__ffs(lefts) - 1u : lane;
    const uint32_t rsrc = split ? (uint32_t)__ffs(run & ~lefts) - 1u : lane;
    __syncwarp();
    if (split) {
      sh.lo[to] = lo;
      sh.hi[to] = hi;
      sh.centre[to] = c;
    }
    const uint32_t m = tk.begin + n_left;
    const bool now_left = lane < s + n_left;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t bl = __shfl_sync(all, cmn[k], lsrc), br = __shfl_sync(all, cmn[k], rsrc);
      const uint32_t tl = __shfl_sync(all, cmx[k], lsrc), tr = __shfl_sync(all, cmx[k], rsrc);
      if (split) {
        tk.box[k] = ordered_to_float(now_left ? bl : br);
        tk.box[3 + k] = ordered_to_float(now_left ? tl : tr);
      }
    }
    if (split) {
      tk.loc = kTemp | (2u * (m - 1u) + (now_left ? 0u : 1u));
      tk.depth += 1u;
      if (now_left) {
        tk.end = m;
        e = s + n_left;
      } else {
        tk.begin = m;
        s += n_left;
      }
    } else {
      open = false;
    }
  }
  __syncwarp();
  if (valid) p.idx_a[pos] = __float_as_uint(sh.hi[lane].w);
  __syncwarp();
}

// ------------------------------------------------------------------ level scan + emit
__device__ __forceinline__ uint64_t children_value(const Decision& d, const Task& tk, uint32_t sub_max) {
  if (!d.split) return 0;
  const uint32_t ws = tk.end - tk.begin;
  const uint32_t nl = d.n_left, nr = ws - d.n_left;
  const uint64_t large = (uint64_t)(nl > sub_max) + (uint64_t)(nr > sub_max);
  return (large << 32) | (uint64_t)(2u - (uint32_t)large);
}

__device__ __forceinline__ Task level_task(const Level& lv, uint32_t t) { return ld_task(lv.large + t); }

template <class T>
__device__ __forceinline__ T block_scan_incl(T v, T* s_warp, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = kLargeBlock / 32;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  if (warp == 0) {
    T w = lane < NW ? s_warp[lane] : (T)0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T n = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += n;
    }
    if (lane < NW) s_warp[lane] = w;
  }
  __syncthreads();
  T prefix = warp > 0 ? s_warp[warp - 1] : (T)0;
  T tt = s_warp[NW - 1];
  __syncthreads();
  *total = tt;
  return v + prefix;
}

// Block b's contiguous segment of the level's tasks.
__device__ __forceinline__ void segment(uint32_t N, uint32_t& lo, uint32_t& hi) {
  const uint32_t seg = (N + gridDim.x - 1) / gridDim.x;
  lo = min(N, blockIdx.x * seg);
  hi = min(N, lo + seg);
}

// Children values of the segment: exclusive scan within the segment
// (scan_vals) and the segment total (scan_sums[block]).
__device__ void scan_segment(const SahParams& p, const Level& lv, SahShared& sh) {
  uint32_t lo, hi;
  segment(lv.L, lo, hi);
  uint64_t carry = 0;
  for (uint32_t base = lo; base < hi; base += kLargeBlock) {
    const uint32_t t = base + threadIdx.x;
    uint64_t v = 0;
    if (t < hi) v = children_value(ld_dec(p.dec + t), level_task(lv, t), p.sub_max);
    uint64_t total;
    const uint64_t incl = block_scan_incl<uint64_t>(v, sh.scan, &total);
    if (t < hi) p.scan_vals[t] = carry + incl - v;
    carry += total;
  }
  if (threadIdx.x == 0) p.scan_sums[blockIdx.x] = carry;
}

// Node numbering (breadth first), the next level's task list and the
// subtree list.
__device__ void emit_children(const SahParams& p, const Level& lv, const Decision& d, const Task& tk, uint64_t ex) {
  uint32_t li = (uint32_t)(ex >> 32), si = (uint32_t)(ex & 0xffffffffu);
  const uint32_t child = lv.node_base + li + si;
  DAabb nd = load_aabb_cg(p.nodes + tk.node);
  nd.left_first = (int32_t)child;
  nd.count = -1;
  store_aabb(p.nodes + tk.node, nd);
  DAabb lb, rb;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lb.min[k] = d.lbox[k];
    lb.max[k] = d.lbox[3 + k];
    rb.min[k] = d.rbox[k];
    rb.max[k] = d.rbox[3 + k];
  }
  lb.count = rb.count = 0;
  lb.left_first = rb.left_first = 0;
  store_aabb(p.nodes + child, lb);
  store_aabb(p.nodes + child + 1, rb);
  const Task lt{child, tk.begin, tk.begin + d.n_left, tk.depth + 1};
  const Task rt{child + 1, tk.begin + d.n_left, tk.end, tk.depth + 1};
  if (lt.end - lt.begin > p.sub_max) lv.large_next[li++] = lt;
  else p.subs[lv.sub_base + si++] = lt;
  if (rt.end - rt.begin > p.sub_max) lv.large_next[li++] = rt;
  else p.subs[lv.sub_base + si++] = rt;
  if (max(d.n_left, tk.end - tk.begin - d.n_left) > (uint32_t)kChunk) p.cnt->big[lv.next_parity] = 1u;
}

__device__ void emit_segment(const SahParams& p, const Level& lv, SahShared& sh, bool advance) {
  // prefix of the block totals before this block, and the level total
  uint64_t before = 0, all = 0;
  for (uint32_t b = threadIdx.x; b < gridDim.x; b += kLargeBlock) {
    const uint64_t v = __ldcg(p.scan_sums + b);
    all += v;
    if (b < blockIdx.x) before += v;
  }
  uint64_t t0, t1;
  block_scan_incl<uint64_t>(before, sh.scan, &t0);
  block_scan_incl<uint64_t>(all, sh.scan, &t1);
  before = t0;
  all = t1;
  uint32_t lo, hi;
  segment(lv.L, lo, hi);
  for (uint32_t t = lo + threadIdx.x; t < hi; t += kLargeBlock) {
    const Decision d = ld_dec(p.dec + t);
    if (d.split) emit_children(p, lv, d, level_task(lv, t), __ldcg(p.scan_vals + t) + before);
  }
  if (advance && blockIdx.x == 0 && threadIdx.x == 0) {
    const uint32_t nl = (uint32_t)(all >> 32), ns = (uint32_t)(all & 0xffffffffu);
    p.cnt->node_count = lv.node_base + nl + ns;
    p.cnt->large = nl;
    p.cnt->sub = lv.sub_base + ns;
  }
}

// Scan and emission of a level of few tasks by one block.
constexpr uint32_t kFewTasks = 4u * kLargeBlock;
__device__ void scan_emit_block(const SahParams& p, const Level& lv, SahShared& sh, bool advance) {
  uint64_t carry = 0;
  for (uint32_t base = 0; base < lv.L; base += kLargeBlock) {
    const uint32_t t = base + threadIdx.x;
    Decision d;
    d.split = 0;
    Task tk{0u, 0u, 0u, 0u};
    if (t < lv.L) {
      d = ld_dec(p.dec + t);
      tk = level_task(lv, t);
    }
    const uint64_t v = t < lv.L ? children_value(d, tk, p.sub_max) : 0ull;
    uint64_t total;
    const uint64_t incl = block_scan_incl<uint64_t>(v, sh.scan, &total);
    if (d.split) emit_children(p, lv, d, tk, carry + incl - v);
    carry += total;
  }
  if (threadIdx.x == 0) {
    const uint32_t nl = (uint32_t)(carry >> 32), ns = (uint32_t)(carry & 0xffffffffu);
    if (advance) {
      p.cnt->node_count = lv.node_base + nl + ns;
      p.cnt->large = nl;
      p.cnt->sub = lv.sub_base + ns;
    } else {
      p.cnt->next_large = nl;
      p.cnt->next_sub = ns;
    }
  }
}

// Blocks take partition chunks in ticket order until all are done.
__device__ void large_partition_phase(const SahParams& p, const Level& lv, uint32_t chunks, SahShared& sh) {
  for (;;) {
    if (threadIdx.x == 0) sh.chunk = atomicAdd(&p.cnt->ticket, 1u);
    __syncthreads();
    const uint32_t c = sh.chunk;
    __syncthreads();
    if (c >= chunks) break;
    large_partition_chunk(p, lv, c, sh);
  }
}

__device__ __forceinline__ Level read_level(const SahParams& p, uint32_t level) {
  Level lv;
  lv.L = __ldcg(&p.cnt->large);
  lv.node_base = __ldcg(&p.cnt->node_count);
  lv.sub_base = __ldcg(&p.cnt->sub);
  lv.large = p.large[level & 1];
  lv.large_next = p.large[(level + 1) & 1];
  lv.parity = level & 1;
  lv.next_parity = (level + 1) & 1;
  lv.src = lv.parity ? p.idx_b : p.idx_a;
  lv.dst = lv.parity ? p.idx_a : p.idx_b;
  return lv;
}

// The breadth-first part of the build: one cooperative launch, the levels of
// the tree one after another, phases separated by grid barriers. Level l
// reads task list large[l & 1] and writes the other one. What bounds it is the
// number of barriers (about 5 us each with the dependent reads around them):
// tasks of at most a chunk are done whole by a block or, up to kTaskWarp
// primitives, a warp, so a level of such tasks needs no binning and partition
// phases, and a level of few tasks is numbered by block 0 alone -- two
// barriers instead of six. 6,400 triangles 397 -> 220 us (12 levels); a warp for
// tasks of up to 256 instead of 64 costs 10 us there.
__global__ void __launch_bounds__(kLargeBlock, 2) k_sah_build(SahParams p) {
  __shared__ SahShared sh;
  const uint32_t G = gridDim.x;
  const uint32_t gwarp = (blockIdx.x * kLargeBlock + threadIdx.x) >> 5, nwarps = G * (kLargeBlock / 32);
  // a level's few tasks go to different blocks first
  const uint32_t spread = (threadIdx.x >> 5) * G + blockIdx.x;
  uint32_t* status = &p.cnt->status;
  for (uint32_t level = 0;; ++level) {
    const Level lv = read_level(p, level);
    const bool big = __ldcg(&p.cnt->big[level & 1]) != 0u;
    if (lv.L == 0) break;
    if (level > kMaxDepth + 1) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(status, kStatusBadIndex);
      break;
    }
    uint32_t chunks = 0;
    if (big) {
      if (blockIdx.x == 0) large_prep(p, lv, sh, kChunk);
      large_bins_init(p, lv);
      if (!grid_sync(p.bar, G, status)) return;
      chunks = __ldcg(&p.cnt->chunks);
      for (uint32_t c = blockIdx.x; c < chunks; c += G) large_bin_chunk(p, lv, c, sh);
      if (!grid_sync(p.bar, G, status)) return;
    }
    for (uint32_t t = blockIdx.x; t < lv.L; t += G) {  // the same tasks for every thread of the block
      const Task tk = ld_task(lv.large + t);
      const uint32_t ws = tk.end - tk.begin;
      if (ws > kTaskWarp && ws <= (uint32_t)kChunk) large_task_block(p, lv, t, sh);
    }
    for (uint32_t t = nwarps > lv.L ? spread : gwarp; t < lv.L; t += nwarps) {
      const Task tk = ld_task(lv.large + t);
      const uint32_t ws = tk.end - tk.begin;
      if (ws > (uint32_t)kChunk) large_decide(p, lv, t, sh);
      else if (ws <= kTaskWarp) large_task_warp(p, lv, t, sh);
    }
    if (!grid_sync(p.bar, G, status)) return;
    if (big) {
      // large partitions (chunks in ticket order)
      large_partition_phase(p, lv, chunks, sh);
      if (!grid_sync(p.bar, G, status)) return;
      for (uint32_t c = blockIdx.x * kLargeBlock + threadIdx.x; c < chunks; c += G * kLargeBlock)
        p.chunk_status[c] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) p.cnt->big[level & 1] = 0u;  // the level after the next sets it again
    if (lv.L <= kFewTasks) {
      if (blockIdx.x == 0) scan_emit_block(p, lv, sh, true);
    } else {
      scan_segment(p, lv, sh);
      if (!grid_sync(p.bar, G, status)) return;
      emit_segment(p, lv, sh, true);
    }
    if (!grid_sync(p.bar, G, status)) return;
  }
}

// Dynamic shared memory of a per-phase launch, sized to the prefix of
// SahShared that the phase uses.
__device__ __forceinline__ SahShared& dyn_shared() {
  extern __shared__ __align__(16) unsigned char sah_dyn[];
  return *reinterpret_cast<SahShared*>(sah_dyn);
}

// ---- the same phases as separate launches (large builds): the level number
// selects the task lists, counters are read at kernel start.
__global__ void __launch_bounds__(kLargeBlock) k_ph_prep(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  if (lv.L == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) p.cnt->chunks = 0;
    return;
  }
  if (blockIdx.x == 0) large_prep(p, lv, sh, 1u);
  large_bins_init(p, lv);
}
// (three blocks per SM: 80 registers; two or four are 1 and 3 % slower at 4M)
__global__ void __launch_bounds__(kLargeBlock, 3) k_ph_bin(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  const uint32_t chunks = __ldcg(&p.cnt->chunks);
  for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) large_bin_chunk(p, lv, c, sh);
}
__global__ void __launch_bounds__(kLargeBlock) k_ph_decide(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  const uint32_t gwarp = (blockIdx.x * kLargeBlock + threadIdx.x) >> 5, nwarps = gridDim.x * (kLargeBlock / 32);
  for (uint32_t t = gwarp; t < lv.L; t += nwarps) large_decide(p, lv, t, sh);
}
__global__ void __launch_bounds__(kLargeBlock) k_ph_partition(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  large_partition_phase(p, lv, __ldcg(&p.cnt->chunks), sh);
}
// Chunk status cleared for the next level, and the numbering of a level: by one
// more block for few tasks, else by the kernels below.
__global__ void __launch_bounds__(kLargeBlock) k_ph_number(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  const uint32_t chunks = __ldcg(&p.cnt->chunks);
  if (lv.L == 0) return;
  if (blockIdx.x + 1u < gridDim.x) {
    for (uint32_t c = blockIdx.x * kLargeBlock + threadIdx.x; c < chunks; c += (gridDim.x - 1u) * kLargeBlock)
      p.chunk_status[c] = 0;
  } else if (lv.L <= kFewTasks) {
    scan_emit_block(p, lv, sh, false);
  }
}
__global__ void __launch_bounds__(kLargeBlock) k_ph_scan(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  if (lv.L > kFewTasks) scan_segment(p, lv, sh);
}
__global__ void __launch_bounds__(kLargeBlock) k_ph_emit(SahParams p, uint32_t level) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  if (lv.L > kFewTasks) emit_segment(p, lv, sh, false);
}
// Counters of the next level (after every block of the kernels before read
// them).
__global__ void __launch_bounds__(kLargeBlock) k_ph_advance(SahParams p, uint32_t level, uint32_t blocks) {
  SahShared& sh = dyn_shared();
  const Level lv = read_level(p, level);
  __syncthreads();  // thread 0 overwrites below what every warp has to read here
  if (lv.L == 0) return;
  if (lv.L <= kFewTasks) {
    if (threadIdx.x == 0) {
      p.cnt->node_count = lv.node_base + p.cnt->next_large + p.cnt->next_sub;
      p.cnt->large = p.cnt->next_large;
      p.cnt->sub = lv.sub_base + p.cnt->next_sub;
    }
    return;
  }
  uint64_t all = 0;
  for (uint32_t b = threadIdx.x; b < blocks; b += kLargeBlock) all += __ldcg(p.scan_sums + b);
  uint64_t tot;
  block_scan_incl<uint64_t>(all, sh.scan, &tot);
  if (threadIdx.x == 0) {
    const uint32_t nl = (uint32_t)(tot >> 32), ns = (uint32_t)(tot & 0xffffffffu);
    p.cnt->node_count = lv.node_base + nl + ns;
    p.cnt->large = nl;
    p.cnt->sub = lv.sub_base + ns;
  }
}

// ---- subtrees and their placement
enum SubPass { kSubWhole, kSubSplit, kSubRest };
template <int PASS>
__global__ void __launch_bounds__(kSubBlock) k_sub_build(SahParams p) {
  extern __shared__ __align__(16) unsigned char sub_dyn[];
  SubShared& sh = reinterpret_cast<SubShared*>(sub_dyn)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t S = PASS == kSubRest ? min(__ldcg(&p.cnt->mid), p.mid_cap) : __ldcg(&p.cnt->sub);
  uint32_t* const head = PASS == kSubRest ? &p.cnt->mid_head : &p.cnt->sub_head;
  SmallList list(p.tiny, p.small_cap, &p.cnt->tiny);  // lane 0's
  MidList mids(p.mid, p.mid_cap, &p.cnt->mid);
  for (;;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(head, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= S) break;
    SubTask root;
    if (PASS == kSubRest) {
      root = reinterpret_cast<const SubTask*>(p.mid)[t];
      if (root.end == 0u) continue;
    } else {
      root = sub_root(p, ld_task(p.subs + t));
    }
    sub_warp_tree<PASS == kSubSplit>(p, root, sh, list, mids);
  }
  if (lane == 0) {
    list.finish();
    if (PASS == kSubSplit) mids.finish();
  }
}

// The listed subtrees of at most kSmall primitives: a warp takes 32 entries at a
// time and builds as many of them side by side as fit its lanes.
__global__ void __launch_bounds__(kSubBlock) k_sub_small(SahParams p) {
  __shared__ SmallShared sh[kSubBlock / 32];
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t all = 0xffffffffu;
  const uint32_t T = min(__ldcg(&p.cnt->tiny), p.small_cap);
  const SubTask* list = reinterpret_cast<const SubTask*>(p.tiny);
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&p.cnt->tiny_head, 32u);
    base = __shfl_sync(all, base, 0);
    if (base >= T) break;
    SubTask mine = {};
    if (base + lane < T) mine = list[base + lane];
    uint32_t size = mine.end - mine.begin;
    if (size > kSmall) {
      atomicOr(&p.cnt->status, kStatusBadIndex);
      size = 0;
    }
    uint32_t incl = size;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(all, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    const uint32_t total = __shfl_sync(all, incl, 31);
    for (uint32_t done = 0; done < total;) {
      // the entries after the first `done` primitives that fit 32 lanes
      const bool in = size > 0u && incl > done && incl <= done + 32u;
      SmallShared& own = sh[threadIdx.x >> 5];
      if (in) own.entry[incl - size - done] = (uint8_t)lane;
      __syncwarp();
      const uint32_t starts = __reduce_or_sync(all, in ? 1u << (incl - size - done) : 0u);
      const uint32_t used = __reduce_max_sync(all, in ? incl : done) - done;
      const uint32_t first = 31u - __clz(starts & (all >> (31u - lane)));  // start of the lane's entry
      const uint32_t src = own.entry[first];
      SubTask tk;
      tk.loc = __shfl_sync(all, mine.loc, src);
      tk.begin = __shfl_sync(all, mine.begin, src);
      tk.end = __shfl_sync(all, mine.end, src);
      tk.depth = __shfl_sync(all, mine.depth, src);
#pragma unroll
      for (int k = 0; k < 6; ++k) tk.box[k] = __shfl_sync(all, mine.box[k], src);
      small_subtrees(p, own, lane < used, tk, first);
      done += used;
    }
  }
}

constexpr uint32_t kScanTile = 4096;  // split positions per tile: 1024 threads x 4

__global__ void __launch_bounds__(1024) k_tile_sums(const uint32_t* __restrict__ flag, uint32_t n,
                                                    uint32_t* __restrict__ tile_off) {
  __shared__ uint32_t s_warp[32];
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * 4u;
  uint32_t v = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k)
    if (base + k < n) v += flag[base + k];
  uint32_t total;
  block_inclusive_scan<1024>(v, s_warp, &total);
  if (threadIdx.x == 0) tile_off[blockIdx.x] = total;
}

// Exclusive offsets of the tiles (one block); the total is the number of
// splits inside the subtrees.
__global__ void __launch_bounds__(1024) k_tile_scan(uint32_t* __restrict__ tile_off, uint32_t tiles, Counters* cnt) {
  __shared__ uint32_t s_warp[32];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < tiles; base += 1024) {
    const uint32_t t = base + threadIdx.x;
    const uint32_t v = t < tiles ? tile_off[t] : 0u;
    uint32_t total;
    const uint32_t incl = block_inclusive_scan<1024>(v, s_warp, &total);
    if (t < tiles) tile_off[t] = carry + incl - v;
    carry += total;
  }
  if (threadIdx.x == 0) cnt->sub_splits = carry;
}

__global__ void __launch_bounds__(1024) k_rank(const uint32_t* __restrict__ flag, uint32_t n,
                                               const uint32_t* __restrict__ tile_off, uint32_t* __restrict__ rank) {
  __shared__ uint32_t s_warp[32];
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * 4u;
  uint32_t f[4], v = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    f[k] = base + k < n ? flag[base + k] : 0u;
    v += f[k];
  }
  uint32_t total;
  uint32_t x = block_inclusive_scan<1024>(v, s_warp, &total) - v + tile_off[blockIdx.x];
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    if (base + k < n) rank[base + k] = x;
    x += f[k];
  }
}

// The node pair of subtree split m goes to top + 2 rank[m] (top: the nodes
// of the breadth-first part); interior nodes get their children's final
// index.
__global__ void __launch_bounds__(kLargeBlock) k_relocate(SahParams p) {
  const uint32_t m = blockIdx.x * kLargeBlock + threadIdx.x;
  if (m == 0 || m >= p.n || !p.sflag[m]) return;
  const uint32_t top = __ldcg(&p.cnt->node_count);
  const uint32_t pair = top + 2u * p.srank[m];
  if (pair + 1u >= 2u * p.n - 1u) {  // past the 2n - 1 nodes
    atomicOr(&p.cnt->status, kStatusBadIndex);
    return;
  }
#pragma unroll
  for (uint32_t k = 0; k < 2; ++k) {
    DAabb nd = load_aabb(p.tnodes + 2u * (m - 1u) + k);
    if (nd.count < 0) {
      const uint32_t c = (uint32_t)nd.left_first;
      if (c == 0 || c >= p.n) {
        atomicOr(&p.cnt->status, kStatusBadIndex);
        return;
      }
      nd.left_first = (int32_t)(top + 2u * p.srank[c]);
    }
    store_aabb(p.nodes + pair + k, nd);
  }
}

// Subtree roots (nodes of the breadth-first part) that split.
__global__ void __launch_bounds__(kLargeBlock) k_fix_roots(SahParams p) {
  const uint32_t S = __ldcg(&p.cnt->sub), top = __ldcg(&p.cnt->node_count);
  for (uint32_t t = blockIdx.x * kLargeBlock + threadIdx.x; t < S && t < p.n + 1u; t += gridDim.x * kLargeBlock) {
    const Task tk = p.subs[t];
    DAabb nd = load_aabb(p.nodes + tk.node);
    if (nd.count >= 0) continue;
    const uint32_t c = (uint32_t)nd.left_first;
    if (c == 0 || c >= p.n) {
      atomicOr(&p.cnt->status, kStatusBadIndex);
      continue;
    }
    nd.left_first = (int32_t)(top + 2u * p.srank[c]);
    store_aabb(p.nodes + tk.node, nd);
  }
}


__global__ void k_sah_init(SahParams p, const DAabb* world) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < p.n) p.idx_a[i] = i;
  if (i == 0) {
    store_aabb(p.nodes, *world);
    const Task root{0u, 0u, p.n, 0u};
    if (p.n > p.sub_max) {
      p.large[0][0] = root;
      p.cnt->large = 1;
      p.cnt->sub = 0;
    } else {
      p.subs[0] = root;
      p.cnt->large = 0;
      p.cnt->sub = 1;
    }
    p.cnt->node_count = 1;
    p.cnt->big[0] = p.n > (uint32_t)kChunk ? 1u : 0u;
    p.cnt->big[1] = 0u;
    p.cnt->status = 0;
    p.cnt->chunks = 0;
    p.cnt->ticket = 0;
    p.cnt->sub_head = 0;
    p.cnt->sub_splits = 0;
    p.cnt->tiny = 0;
    p.cnt->tiny_head = 0;
    p.cnt->mid = 0;
    p.cnt->mid_head = 0;
  }
}

}  // namespace

ResultCode build_binned_sah(const DAabb* aabbs, const float4* centers, size_t n_, size_t prims_per_leaf,
                            cudaStream_t s, BuildOutput* out) {
  if (n_ == 0) return NoPrimitives;
  if (n_ >= (1u << 30)) return InvalidArgument;
  const uint32_t n = (uint32_t)n_;
  const uint32_t node_cap = 2u * n - 1u;
  cudaError_t e;
  DAabb* nodes = nullptr;
  uint32_t* indices = nullptr;
  if ((e = device_alloc(&nodes, node_cap, s))) return cuda_rc(e);
  if ((e = device_alloc(&indices, n, s))) {
    pool_free(nodes, s);
    return cuda_rc(e);
  }
  auto fail = [&](ResultCode rc) {
    pool_free(nodes, s);
    pool_free(indices, s);
    return rc;
  };
  // The breadth-first part of builds up to kCoopMaxPrims runs as one
  // cooperative launch: the middle levels hold many small tasks, so the grid
  // covers every SM, with one block each for small builds, whose time is the
  // barriers', and the full resident grid above (builds with both trees, one
  // block against two: 20k triangles 723 / 780 us, 100k 1,217 / 1,176, 400k
  // 2,047 / 1,887). Large builds launch the phases separately, which lets each
  // phase run at its own occupancy, and read the counts back every fourth
  // level; cooperative against that, us: 1.2M 3,225 / 3,426, 1.6M 3,815 / 3,956,
  // 2M 4,470 / 4,507, 3M 7,060 / 6,980, 4M 8,050 / 7,845.
  const bool coop = n <= kCoopMaxPrims;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, coop ? (const void*)k_sah_build
                                                                         : (const void*)k_ph_partition,
                                                         kLargeBlock, coop ? 0 : kShChunk)))
    return fail(cuda_rc(e));
  if (per_sm < 1) return fail(DeviceError);
  const uint32_t grid = (uint32_t)sm_count() * (coop && n <= 65536u ? 1u : (uint32_t)per_sm);
  uint32_t sub_max = n / 2048u;
  sub_max = sub_max < 32u ? 32u : (sub_max > kWarpMax ? kWarpMax : sub_max);
  const uint32_t large_cap = n / (sub_max + 1) + 2;
  const uint32_t sub_cap = n + 1;
  const uint32_t chunk_cap = n / kChunk + large_cap + 2;
  const uint32_t tiles = (n + kScanTile - 1) / kScanTile;
  int sub_per_sm = 0;
  const size_t sub_smem = (kSubBlock / 32) * sizeof(SubShared);
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sub_per_sm, k_sub_build<kSubWhole>, kSubBlock, sub_smem)))
    return fail(cuda_rc(e));
  if (sub_per_sm < 1) return fail(DeviceError);
  uint32_t sub_grid = (uint32_t)sm_count() * (uint32_t)sub_per_sm;
  const uint32_t want = (n / (sub_max > 8u ? 8u : sub_max) + kSubBlock / 32) / (kSubBlock / 32) + 1u;
  if (want < sub_grid) sub_grid = want;
  // listed subtrees hold a primitive or more; every warp may leave a chunk
  const bool two_launches = sub_max > kMidFrom;
  const uint32_t sub_warps = sub_grid * (kSubBlock / 32);
  const uint32_t small_cap = n + sub_warps * kListChunk * (two_launches ? 2u : 1u);
  const uint32_t mid_cap = two_launches ? n / (kSmall + 1u) + sub_warps * kMidChunk : 0u;
  constexpr size_t kBarWords = (sizeof(GridBarrier) + 3) / 4;
  const size_t zero_words = kBarWords + chunk_cap + n;
  ScratchPack scratch;
  DAabb *world, *tnodes;
  uint32_t *acc, *idx_b, *bins, *chunk_base, *zeros, *srank, *tile_off;
  Task *large0, *large1, *subs;
  SubTask *tiny, *mid;
  Decision* dec;
  float* tbox;
  uint64_t *scan_vals, *scan_sums;
  Counters* cnt;
  scratch.add(&world, 1);
  scratch.add(&acc, kBoundsWords);
  scratch.add(&idx_b, n);
  scratch.add(&bins, (size_t)large_cap * kTaskBinWords);
  scratch.add(&chunk_base, large_cap + 1);
  scratch.add(&zeros, zero_words);  // barrier, chunk status, split flags
  scratch.add(&large0, large_cap);
  scratch.add(&large1, large_cap);
  scratch.add(&subs, sub_cap);
  scratch.add(&dec, large_cap);
  scratch.add(&tbox, (size_t)large_cap * 6);
  scratch.add(&scan_vals, large_cap);
  scratch.add(&scan_sums, grid);
  scratch.add(&cnt, 1);
  scratch.add(&tnodes, 2 * (size_t)n);
  scratch.add(&srank, n);
  scratch.add(&tile_off, tiles + 1);
  scratch.add(&tiny, small_cap);
  scratch.add(&mid, mid_cap);
  if ((e = scratch.alloc(s)) || (e = cudaMemsetAsync(zeros, 0, zero_words * 4, s))) return fail(cuda_rc(e));
  uint32_t* const chunk_status = zeros + kBarWords;
  uint32_t* const sflag = chunk_status + chunk_cap;
  if ((e = launch_world_bounds(aabbs, n, world, acc, s))) return fail(cuda_rc(e));

  SahParams p;
  p.aabbs = aabbs;
  p.centers = centers;
  p.nodes = nodes;
  p.idx_a = indices;
  p.idx_b = idx_b;
  p.n = n;
  p.sub_max = sub_max;
  p.max_leaf = prims_per_leaf == 0 ? 1u : (uint32_t)(prims_per_leaf > 0xffffffffu ? 0xffffffffu : prims_per_leaf);
  p.large[0] = large0;
  p.large[1] = large1;
  p.subs = subs;
  p.tiny = tiny;
  p.small_cap = small_cap;
  p.mid = mid;
  p.mid_cap = mid_cap;
  p.dec = dec;
  p.tbox = tbox;
  p.bins = bins;
  p.chunk_base = chunk_base;
  p.chunk_status = chunk_status;
  p.scan_vals = scan_vals;
  p.scan_sums = scan_sums;
  p.tnodes = tnodes;
  p.sflag = sflag;
  p.srank = srank;
  p.tile_off = tile_off;
  p.cnt = cnt;
  p.bar = reinterpret_cast<GridBarrier*>(zeros);
  k_sah_init<<<(n + 255) / 256, 256, 0, s>>>(p, world);
  Counters h{};
  if (n > sub_max) {
    if (coop) {
      // the subtree stage below reads the counts it needs on the device
      void* args[] = {&p};
      if ((e = cudaLaunchCooperativeKernel((void*)k_sah_build, dim3(grid), dim3(kLargeBlock), args, 0, s)))
        return fail(cuda_rc(e));
    } else {
      // The kernels read a level's counts on the device and do nothing past
      // the last one, so the host looks at them every fourth level only.
      h.large = 1u;
      int bin_per_sm = 0;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bin_per_sm, k_ph_bin, kLargeBlock, kShBins)))
        return fail(cuda_rc(e));
      const uint32_t sms = (uint32_t)sm_count(), bin_grid = sms * (uint32_t)(bin_per_sm < 1 ? 1 : bin_per_sm);
      for (uint32_t level = 0; h.large > 0;) {
        if (level > kMaxDepth + 1) return fail(Error);
        for (uint32_t k = 0; k < 4; ++k, ++level) {
          k_ph_prep<<<sms, kLargeBlock, kShSmall, s>>>(p, level);
          k_ph_bin<<<bin_grid, kLargeBlock, kShBins, s>>>(p, level);
          k_ph_decide<<<sms * 2u, kLargeBlock, kShBins, s>>>(p, level);
          k_ph_partition<<<grid, kLargeBlock, kShChunk, s>>>(p, level);
          k_ph_number<<<9, kLargeBlock, kShSmall, s>>>(p, level);
          if (large_cap > kFewTasks) {  // else no level has that many tasks
            k_ph_scan<<<grid, kLargeBlock, kShSmall, s>>>(p, level);
            k_ph_emit<<<grid, kLargeBlock, kShSmall, s>>>(p, level);
          }
          k_ph_advance<<<1, kLargeBlock, kShSmall, s>>>(p, level, grid);
        }
        if ((e = cudaGetLastError())) return fail(cuda_rc(e));
        if ((e = cudaMemcpyAsync(&h, cnt, sizeof(Counters), cudaMemcpyDeviceToHost, s)) ||
            (e = cudaStreamSynchronize(s)))
          return fail(cuda_rc(e));
        if (h.status) break;
      }
    }
    if (h.status) return fail(h.status & kStatusTimeout ? Timeout : Error);
    if (h.large > 0) return fail(Error);
  }
  // subtrees, then their node pairs after the breadth-first part (the
  // kernels read the subtree count and the breadth-first node count on the
  // device)
  {
    if (two_launches) {
      k_sub_build<kSubSplit><<<sub_grid, kSubBlock, sub_smem, s>>>(p);
      k_sub_build<kSubRest><<<sub_grid, kSubBlock, sub_smem, s>>>(p);
    } else {
      k_sub_build<kSubWhole><<<sub_grid, kSubBlock, sub_smem, s>>>(p);
    }
    int small_per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&small_per_sm, k_sub_small, kSubBlock, 0)))
      return fail(cuda_rc(e));
    const uint32_t small_grid = (uint32_t)sm_count() * (uint32_t)(small_per_sm < 1 ? 1 : small_per_sm);
    const uint32_t small_want = (small_cap / 32u + kSubBlock / 32) / (kSubBlock / 32);
    k_sub_small<<<small_want < small_grid ? small_want : small_grid, kSubBlock, 0, s>>>(p);
    k_tile_sums<<<tiles, 1024, 0, s>>>(sflag, n, tile_off);
    k_tile_scan<<<1, 1024, 0, s>>>(tile_off, tiles, cnt);
    k_rank<<<tiles, 1024, 0, s>>>(sflag, n, tile_off, srank);
    k_relocate<<<(n + kLargeBlock - 1) / kLargeBlock, kLargeBlock, 0, s>>>(p);
    const unsigned fix_blocks = (unsigned)((n + kLargeBlock) / kLargeBlock);
    k_fix_roots<<<fix_blocks < (unsigned)sm_count() * 4u ? fix_blocks : (unsigned)sm_count() * 4u, kLargeBlock, 0,
                  s>>>(p);
    if ((e = cudaGetLastError())) return fail(cuda_rc(e));
    if ((e = cudaMemcpyAsync(&h, cnt, sizeof(Counters), cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
      return fail(cuda_rc(e));
    if (h.status) return fail(h.status & kStatusTimeout ? Timeout : Error);
    if (h.large > 0) return fail(Error);  // the breadth-first part did not finish
  }
  const uint64_t total = (uint64_t)h.node_count + 2ull * h.sub_splits;
  if (total > node_cap) return fail(Error);
  out->nodes = nodes;
  out->indices = indices;
  out->node_count = (uint32_t)total;
  return Ok;
}

}  // namespace rtbvh
