// BVH2 -> 4-wide MBVH collapse (Mbvh::construct, src/bvh.rs:381-404, and
// MbvhNode::merge_nodes, src/mbvh_node.rs:297-411) on the GPU.
//
// The reference numbers quad nodes by a recursive walk that hands out
// `pool_ptr++` in slot order (a pre-order over quad nodes). Quad nodes are
// exactly the interior BVH2 nodes at even depth, and the quad subtree rooted
// at such a node g holds cntE(g) quad nodes, where
//   cntE(c) = 1 + cntO(left) + cntO(right),  cntO(c) = cntE(left) + cntE(right)
// for interior c and 0 for leaves. So:
//   1. parent pointers;
//   2. cntE/cntO bottom-up (the second child to arrive at a parent computes it);
//   3. every quad node's index from the counts on its way up (find_place):
//      no order between levels;
//   4. the quad nodes, one thread each in index order.
// The slot contents reproduce merge_nodes line by line, including its quirks
// (a leaf child keeps the parent's box in its slot; the second slot of that
// side stays empty with the parent's box).
#include <mutex>

#include "lib_internal.h"

namespace rtbvh {

namespace {

constexpr int kBlock = 256;
constexpr uint32_t kNone = 0xffffffffu;

// Arrival at a parent in the bottom-up walks that hand on boxes: atomic add
// with acquire and release semantics at device scope. The release publishes
// this thread's writes for its child; the second arrival's acquire makes the
// sibling's writes visible to it (one instruction where fence + add + fence
// were).
__device__ __forceinline__ uint32_t arrive_acq_rel(uint32_t* p) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
  return old;
}
__device__ __forceinline__ uint64_t add_acq_rel(uint64_t* p, uint64_t v) {
  uint64_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

__device__ __forceinline__ bool box_contains(const DAabb& outer, const DAabb& inner) {
  // false on NaN: such a box counts as not containing
  return outer.min[0] <= inner.min[0] && outer.min[1] <= inner.min[1] && outer.min[2] <= inner.min[2] &&
         outer.max[0] >= inner.max[0] && outer.max[1] >= inner.max[1] && outer.max[2] >= inner.max[2];
}

// Vertex box of triangle p (9 floats), grown by 1e-4: what Bvh::refit
// (src/bvh.rs:176-205) gives a leaf of that one triangle.
__device__ __forceinline__ DAabb grown_triangle_box(const float* __restrict__ vertices, uint32_t p) {
  const float* v = vertices + 9 * (size_t)p;
  DAabb b;
  for (int a = 0; a < 3; ++a) { b.min[a] = 1e34f; b.max[a] = -1e34f; }
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float x = __ldg(v + 3 * j + a);
      b.min[a] = rs_min(b.min[a], x);
      b.max[a] = rs_max(b.max[a], x);
    }
  for (int a = 0; a < 3; ++a) { b.min[a] = b.min[a] - 0.0001f; b.max[a] = b.max[a] + 0.0001f; }
  b.count = 0;
  b.left_first = 0;
  return b;
}

// Parent word of a node: parent << 1 | 1 for the right child of a pair
// (kNone: no parent). Node indices that left_first can name are below 2^31.
__device__ __forceinline__ uint32_t parent_of(uint32_t w) { return w >> 1; }

// The counts of a node in one word, so that the two children of a node add
// theirs to it and the second one to arrive has the sums with no further
// reads: bits 0-29 cntE (an interior node starts with the 1 of its own, a leaf
// with 0), bits 30-59 cntO, bit 60 the node's box does not contain its box from
// the triangles (TRIS), bits 62-63 children arrived (a leaf starts with both).
constexpr uint64_t kArrived = 1ull << 62;
constexpr uint64_t kBadBox = 1ull << 60;
constexpr uint32_t kCountMask = (1u << 30) - 1u;
__device__ __forceinline__ bool counted(uint64_t c) { return (c >> 62) == 2u; }
__device__ __forceinline__ uint32_t cnt_e_of(uint64_t c) { return (uint32_t)c & kCountMask; }
__device__ __forceinline__ uint32_t cnt_o_of(uint64_t c) { return (uint32_t)(c >> 30) & kCountMask; }

// cnt / arrive / known may be NULL.
__global__ void __launch_bounds__(kBlock)
    k_parents(const DAabb* __restrict__ nodes, uint32_t node_count, uint32_t* __restrict__ parent,
              uint32_t* __restrict__ arrive, uint64_t* __restrict__ cnt, uint2* __restrict__ known,
              uint32_t* __restrict__ status) {
  uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= node_count) return;
  DAabb nd = load_aabb(nodes + c);
  if (arrive) arrive[c] = 0;
  if (cnt) cnt[c] = nd.count >= 0 ? 2u * kArrived : 1u;
  if (known) known[c] = make_uint2(kNone, kNone);
  if (nd.count < 0 && nd.left_first >= 0 && c <= 0x7fffffffu) {
    uint32_t lf = (uint32_t)nd.left_first;
    if (lf + 1 < node_count) {
      parent[lf] = c << 1;
      parent[lf + 1] = c << 1 | 1u;
    } else {
      atomicOr(status, kStatusBadIndex);
    }
  }
}

// Sibling of node x with parent word w.
__device__ __forceinline__ uint32_t sibling_of(uint32_t x, uint32_t w) { return (w & 1u) ? x - 1u : x + 1u; }

// Counts, bottom up: the second child to arrive at a parent goes on from
// there. What bounds a walk is one atomic round trip per level; the parent of
// the next level is read meanwhile. Counts of 200k sphere
// triangles 62 -> 22 us, of 1M 111 -> 39 us (before: parent, arrival counter,
// node and both counts one after another); refit walk of 200k 80 -> 53 us.
// Two leaves of a pair in one warp meet by shuffles, without the atomics (and
// with TRIS their fences): 4M clustered triangles (SAH) 558 -> 521 us, 64 meshes
// 187 -> 57. Blocks of 128 and 16 of them per SM (32 registers): a block stays
// until its longest walk ends, mostly with a few lanes, so walks in flight are
// what counts; the 4M build with 256 threads and 38 registers 8,336 us, 256 x 8
// 8,104, 128 x 16 8,072, 64 x 32 8,088.
// With TRIS, the same walk also computes every node's traversal box `tb`
// from the triangles: a leaf's is the union of its triangles' vertex boxes
// grown by 1e-4, an interior node's the union of its children's (the union
// of boxes grown by 1e-4 is the union grown by 1e-4); count/left_first are
// copied from `nodes`.
constexpr int kCountBlock = 128, kCountBlocks = 16;
template <bool TRIS>
__global__ void __launch_bounds__(kCountBlock, kCountBlocks)
    k_counts_bottom_up(const DAabb* __restrict__ nodes, uint32_t node_count, const uint32_t* __restrict__ parent,
                       uint64_t* __restrict__ cnt, MbvhTriangles tri, uint32_t* __restrict__ status) {
  const uint32_t c = blockIdx.x * kCountBlock + threadIdx.x, lane = threadIdx.x & 31u;
  uint32_t w = kNone;
  bool leaf = false;  // walks start at leaves
  DAabb box = {};
  if (c < node_count) {
    w = __ldg(parent + c);
    if (TRIS) box = load_aabb(nodes + c);
    leaf = (TRIS ? box.count : __ldg(&nodes[c].count)) >= 0;
  }
  if (TRIS && leaf) {
    const DAabb nd = box;
    for (int a = 0; a < 3; ++a) { box.min[a] = 1e34f; box.max[a] = -1e34f; }
    if (nd.left_first >= 0) {
      for (int a = 0; a < 3; ++a) { box.min[a] = 1e34f - 0.0001f; box.max[a] = -1e34f + 0.0001f; }
      for (int32_t i = 0; i < nd.count; ++i) {
        const uint32_t slot = (uint32_t)nd.left_first + (uint32_t)i;
        const uint32_t p = slot < tri.index_count ? __ldg(tri.indices + slot) : kNone;
        if (p >= tri.vertex_count) {
          atomicOr(status, kStatusBadIndex);
          break;
        }
        const DAabb t = grown_triangle_box(tri.vertices, p);
        for (int a = 0; a < 3; ++a) { box.min[a] = rs_min(box.min[a], t.min[a]); box.max[a] = rs_max(box.max[a], t.max[a]); }
      }
    }
    store_aabb(tri.tb + c, box);
  }
  uint32_t x = c, e = 0, o = 0;
  // two leaves of one pair: nothing else arrives at their parent
  const uint32_t other = (w & 1u) ? lane - 1u : lane + 1u;
  const uint32_t pair_w = __shfl_sync(0xffffffffu, leaf ? w : kNone, (int)(other & 31u));
  const bool pair = leaf && w != kNone && other < 32u && pair_w == (w ^ 1u);
  if (TRIS) {
    for (int a = 0; a < 3; ++a) {
      const float mn = __shfl_sync(0xffffffffu, box.min[a], (int)(other & 31u));
      const float mx = __shfl_sync(0xffffffffu, box.max[a], (int)(other & 31u));
      if (pair) {
        box.min[a] = rs_min(box.min[a], mn);
        box.max[a] = rs_max(box.max[a], mx);
      }
    }
  }
  if (!leaf || (pair && (w & 1u))) return;
  if (pair) {
    x = parent_of(w);
    uint64_t sum = 2u * kArrived + 1u;
    if (TRIS) {
      const DAabb pn = load_aabb(nodes + x);
      box.count = pn.count;
      box.left_first = pn.left_first;
      store_aabb(tri.tb + x, box);
      if (!box_contains(pn, box)) sum |= kBadBox;
    }
    cnt[x] = sum;
    e = 1;
    w = __ldg(parent + x);
  }
  for (uint32_t steps = 0; steps < node_count; ++steps) {
    if (w == kNone) break;
    const uint32_t p = parent_of(w);
    const uint64_t mine = kArrived | ((uint64_t)e << 30) | (uint64_t)o;  // to cntO and cntE
    DAabb pn;
    if (TRIS) pn = load_aabb(nodes + p);
    const uint32_t above = __ldg(parent + p);
    const uint64_t old = TRIS ? add_acq_rel(cnt + p, mine)
                              : atomicAdd(reinterpret_cast<unsigned long long*>(cnt + p), (unsigned long long)mine);
    if ((old >> 62) != 1u) break;  // the first arrival: the sibling goes on (more than two: no tree)
    const uint64_t sum = old + mine;
    if (TRIS) {
      const DAabb sib = load_aabb_cg(tri.tb + sibling_of(x, w));
      for (int a = 0; a < 3; ++a) {
        box.min[a] = rs_min(box.min[a], sib.min[a]);
        box.max[a] = rs_max(box.max[a], sib.max[a]);
      }
      box.count = pn.count;
      box.left_first = pn.left_first;
      store_aabb(tri.tb + p, box);
      if (!box_contains(pn, box)) atomicAdd(reinterpret_cast<unsigned long long*>(cnt + p), kBadBox);
    }
    e = cnt_e_of(sum);
    o = cnt_o_of(sum);
    x = p;
    w = above;
  }
}

struct CollapseParams {
  const DAabb* nodes;
  uint32_t node_count;
  const uint32_t* parent;  // parent words
  const uint64_t* cnt;
  uint2* known;            // places found so far: {place << 1 | depth parity, nearest bad box}; roots preset
  uint32_t* quads;         // BVH2 node of every quad node
  DMNode* mnodes;
  uint32_t m_total;        // capacity of quads / mnodes / tboxes
  const uint32_t* m_count; // quad nodes (device)
  bool forest;             // several meshes (k_seg_mbase)
  uint32_t* status;
  // escape flags only: triangles, the count of escaped triangles
  MbvhTriangles tri;
  uint32_t* escaped;
  DTBox* tboxes;  // optional (TRIS): subtree boxes of every quad node's slots
};

__device__ __forceinline__ uint2 ld_place(const uint2* p) {
  const unsigned long long v = __ldcg(reinterpret_cast<const unsigned long long*>(p));
  return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
__device__ __forceinline__ void st_place(uint2* p, uint2 v) {
  __stcg(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v.x | ((unsigned long long)v.y << 32));
}

// Place of interior node x: a node at even depth is a quad node and its
// place is its quad index; the quad nodes below a node at odd depth start at
// its place. From parent to child the place grows by
//   even parent: 1 + (right child: cntO(left sibling))
//   odd parent:  (right child: cntE(left sibling)).
// The walk goes up until it meets a node whose place is known (other threads
// publish theirs as they find them; what is not there yet only makes the
// walk longer, nothing waits) and keeps the sums for both parities x may
// have. Only counted nodes are passed: they form trees, so the walk ends.
// What bounds it is the latency of the walk, one dependent read per level;
// nodes near the root have low indices and are placed first, so most walks
// are short. The level-by-level frontier it replaces spent a grid barrier
// per level (collapse of 200k
// sphere triangles 172 us; k_place 27 + k_quads 13 us now; refit of them with
// both trees 824 -> 440 us).
// bad (TRIS): the nearest quad node at or above x whose box misses
// triangles below it (kNone: none).
struct Place {
  uint32_t pos, parity, bad;
  bool ok;
};
template <bool TRIS>
__device__ Place find_place(const CollapseParams& p, uint32_t x) {
  uint32_t even = 0, odd = 0;                 // sums if the current node lies at even / odd depth
  uint32_t bad_even = kNone, bad_odd = kNone;  // the same for the nearest bad quad node
  uint32_t cur = x;
  for (uint32_t k = 0; k < p.node_count; ++k) {
    const uint2 s = ld_place(p.known + cur);
    const uint32_t w = __ldg(p.parent + cur);
    const uint64_t own = __ldg(p.cnt + cur);
    if (s.x != kNone) {
      const bool is_even = (s.x & 1u) == 0u;
      Place r;
      r.pos = (s.x >> 1) + (is_even ? even : odd);
      r.parity = (s.x & 1u) ^ (k & 1u);
      r.bad = is_even ? bad_even : bad_odd;
      if (r.bad == kNone) r.bad = s.y;
      r.ok = true;
      return r;
    }
    if (w == kNone || !counted(own)) break;
    if (TRIS && (own & kBadBox) && bad_even == kNone) bad_even = cur;
    uint32_t e = 0, o = 1u;
    if (w & 1u) {
      const uint64_t sib = __ldg(p.cnt + cur - 1u);
      e = cnt_e_of(sib);
      o += cnt_o_of(sib);
    }
    // cur at even depth: its parent is odd
    const uint32_t se = even + e, so = odd + o, be = bad_even, bo = bad_odd;
    odd = se;
    even = so;
    bad_odd = be;
    bad_even = bo;
    cur = parent_of(w);
  }
  Place r;
  r.pos = r.parity = 0u;
  r.bad = kNone;
  r.ok = false;
  return r;
}

// Four 256-bit stores: neighbouring threads write neighbouring 128-byte
// nodes, so every store fills whole sectors.
__device__ __forceinline__ void store_node(DMNode* out, const DMNode& m) {
  const float* f = reinterpret_cast<const float*>(&m);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(reinterpret_cast<float*>(out) + 8 * k),
                 "f"(f[8 * k]), "f"(f[8 * k + 1]), "f"(f[8 * k + 2]), "f"(f[8 * k + 3]), "f"(f[8 * k + 4]),
                 "f"(f[8 * k + 5]), "f"(f[8 * k + 6]), "f"(f[8 * k + 7])
                 : "memory");
}

__device__ __forceinline__ void set_slot_box(DMNode& m, int i, const DAabb& b) {
  m.min_x[i] = b.min[0]; m.min_y[i] = b.min[1]; m.min_z[i] = b.min[2];
  m.max_x[i] = b.max[0]; m.max_y[i] = b.max[1]; m.max_z[i] = b.max[2];
}

// Escape flags of a quad node's leaf slots (TRIS): a leaf slot's triangle is
// escaped when its vertex box grown by 1e-4 is not inside every slot box on
// the way to it -- the reference's walk tests these boxes before it yields
// the triangle (src/iter_indices.rs:264-313), so it can miss the triangle's
// hits. Those boxes are the leaf's slot box and the boxes of the quad nodes
// on the way up (but the root's, which is no slot). A quad node's box that
// contains its box from the triangles contains every triangle below it, so
// only the others, marked kBadBox, are compared; they are few. Flags go to
// the flags word of each leaf-ordered triangle record (kTriEscape).
__device__ void mark_escapes(const CollapseParams& p, const DMNode& m, uint32_t bad) {
  uint32_t n_esc = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int32_t ch = m.children[i], cnt = m.counts[i];
    if (cnt < 0) continue;  // empty or interior slot
    DAabb slot_box;
    slot_box.min[0] = m.min_x[i]; slot_box.min[1] = m.min_y[i]; slot_box.min[2] = m.min_z[i];
    slot_box.max[0] = m.max_x[i]; slot_box.max[1] = m.max_y[i]; slot_box.max[2] = m.max_z[i];
    for (int32_t j = 0; j < cnt; ++j) {
      const uint32_t slot = (uint32_t)ch + (uint32_t)j;
      const uint32_t prim = slot < p.tri.index_count ? __ldg(p.tri.indices + slot) : kNone;
      if (prim >= p.tri.vertex_count) {
        atomicOr(p.status, kStatusBadIndex);
        break;
      }
      const DAabb t = grown_triangle_box(p.tri.vertices, prim);
      bool inside = box_contains(slot_box, t);
      uint32_t b = bad;
      while (inside && b != kNone) {
        inside = box_contains(load_aabb(p.nodes + b), t);
        // the next one above b: its grandparent's (b lies at even depth >= 2)
        const uint32_t w = __ldg(p.parent + b);
        const uint32_t gw = w != kNone ? __ldg(p.parent + parent_of(w)) : kNone;
        b = gw != kNone ? find_place<true>(p, parent_of(gw)).bad : kNone;
      }
      reinterpret_cast<float*>(p.tri.tris + (size_t)kTriFloat4 * slot + 1)[3] =
          __uint_as_float(inside ? 0u : kTriEscape);
      n_esc += inside ? 0u : 1u;
    }
  }
  if (n_esc) atomicAdd(p.escaped, n_esc);
}

// merge_nodes(mi, c) without the recursion: fills quad node mi.
template <bool TRIS>
__device__ void emit_quad(const CollapseParams& p, uint32_t c, uint32_t mi, uint32_t bad) {
  const DAabb cur = load_aabb(p.nodes + c);
  DMNode m;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    set_slot_box(m, i, cur);
    m.children[i] = -1;
    m.counts[i] = -1;
  }
  int32_t nodes_[4] = {-1, -1, -1, -1};
  int32_t leafs[4] = {-1, -1, -1, -1};
  int32_t sub[4] = {-1, -1, -1, -1};  // BVH2 node under each slot (TRIS: its box from the triangles)
  if (p.forest && cur.count >= 0) {
    // Root leaf of a mesh: the single-mesh tree has this one node, so
    // merge_nodes finds only the root itself in slot 0 (its left_first is
    // no node of this forest).
    nodes_[0] = cur.left_first;
    leafs[0] = cur.count;
  } else if (cur.left_first >= 0) {
    const uint32_t lf = (uint32_t)cur.left_first;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int s0 = 2 * side;
      const uint32_t child = lf + side;
      if (child < p.node_count) {
        const DAabb cn = load_aabb(p.nodes + child);
        if (cn.left_first >= 0) {
          const uint32_t clf = (uint32_t)cn.left_first;
          if (cn.count >= 0) {
            nodes_[s0] = (int32_t)clf;
            leafs[s0] = cn.count;
            sub[s0] = (int32_t)child;
          } else if (clf + 1 < p.node_count) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const DAabb g = load_aabb(p.nodes + clf + k);
              if (g.count >= 0) {
                nodes_[s0 + k] = g.left_first;
                leafs[s0 + k] = g.count;
              } else {
                nodes_[s0 + k] = (int32_t)(clf + k);
              }
              set_slot_box(m, s0 + k, g);
              sub[s0 + k] = (int32_t)(clf + k);
            }
          } else {
            atomicOr(p.status, kStatusBadIndex);
          }
        }
      }
    }
  }
  uint32_t next_index = mi + 1u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int32_t node = nodes_[i];
    const int32_t count = leafs[i];
    if (node >= 0 && count >= 0) {
      m.children[i] = node;
      m.counts[i] = count;
      continue;
    } else if (node < 0) {
      if (node != -1) atomicOr(p.status, kStatusBadIndex);
      continue;
    }
    const uint64_t below = __ldg(p.cnt + node);
    if (next_index < p.m_total && counted(below)) m.children[i] = (int32_t)next_index;
    else atomicOr(p.status, kStatusBadIndex);
    next_index += cnt_e_of(below);
  }
  if (mi < p.m_total) {
    store_node(p.mnodes + mi, m);
    if (TRIS) mark_escapes(p, m, bad);
    if (TRIS && p.tboxes) {
      DTBox t;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        bool ok = sub[i] >= 0 && (uint32_t)sub[i] < p.node_count;
        DAabb b = cur;
        if (ok) b = load_aabb(p.tri.tb + sub[i]);
        for (int a = 0; a < 3; ++a)  // false for NaN
          ok = ok && fabsf(b.min[a]) <= kCompactRange && fabsf(b.max[a]) <= kCompactRange;
        const float inf = __int_as_float(0x7f800000);
        t.min_x[i] = ok ? b.min[0] : -inf; t.max_x[i] = ok ? b.max[0] : inf;
        t.min_y[i] = ok ? b.min[1] : -inf; t.max_y[i] = ok ? b.max[1] : inf;
        t.min_z[i] = ok ? b.min[2] : -inf; t.max_z[i] = ok ? b.max[2] : inf;
      }
      float4* td = reinterpret_cast<float4*>(p.tboxes + mi);
      const float4* ts = reinterpret_cast<const float4*>(&t);
#pragma unroll
      for (int k = 0; k < 6; ++k) td[k] = ts[k];
    }
  } else {
    atomicOr(p.status, kStatusBadIndex);
  }
}

template <bool TRIS>
__global__ void __launch_bounds__(kBlock) k_quads(CollapseParams p) {
  const uint32_t mi = blockIdx.x * kBlock + threadIdx.x;
  if (mi >= min(__ldg(p.m_count), p.m_total)) return;
  const uint32_t c = __ldg(p.quads + mi);
  if (c >= p.node_count) {  // not placed: only after another error
    atomicOr(p.status, kStatusBadIndex);
    return;
  }
  emit_quad<TRIS>(p, c, mi, TRIS ? p.known[c].y : kNone);
}

// The root's place, and the number of quad nodes for the host. A root whose
// count did not come up (no tree) is an error. *bad_root: the root is interior
// and its box misses triangles (kBadBox).
__global__ void k_root_place(const uint64_t* cnt, const DAabb* nodes, uint2* known, uint32_t m_cap, uint32_t* m_total,
                             uint32_t* walloc, uint32_t* bad_root, uint32_t* status) {
  if (threadIdx.x == 0) {
    *walloc = 1u;  // traversal node 0 is the root's
    const uint64_t c = *cnt;
    const uint32_t t = nodes->count < 0 ? cnt_e_of(c) : 1u;
    if (!counted(c) || t == 0u || t > m_cap) atomicOr(status, kStatusBadIndex);
    else *known = make_uint2(0u, kNone);
    *m_total = t;
    *bad_root = (c & kBadBox) ? 1u : 0u;
  }
}

// ---------------------------------------------------------------- many meshes
// A concatenated forest: mesh m's root is BVH2 node 2 off_m - m. Its quad
// nodes get the contiguous index range [mbase[m], mbase[m+1]) (the
// single-mesh numbering shifted by mbase[m]): its root's place is mbase[m],
// and k_quads does the rest for all meshes at once.
__global__ void __launch_bounds__(1024) k_seg_mbase(const DAabb* __restrict__ nodes, const uint64_t* __restrict__ cnt,
                                                    const uint32_t* __restrict__ prim_off, uint32_t mesh_count,
                                                    uint2* __restrict__ known, uint32_t* __restrict__ mbase) {
  __shared__ uint32_t s_warp[32];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < mesh_count; base += 1024) {
    const uint32_t m = base + threadIdx.x;
    uint32_t q = 0;
    if (m < mesh_count) {
      const uint32_t off = prim_off[m], n = prim_off[m + 1] - off;
      if (n > 0) {
        const uint32_t root = 2u * off - m;
        if (counted(cnt[root])) q = load_aabb(nodes + root).count < 0 ? cnt_e_of(cnt[root]) : 1u;
      }
    }
    uint32_t total;
    const uint32_t incl = block_inclusive_scan<1024>(q, s_warp, &total);
    if (m < mesh_count) {
      mbase[m] = carry + incl - q;
      if (q) known[2u * prim_off[m] - m] = make_uint2((carry + incl - q) << 1, kNone);
    }
    carry += total;
  }
  if (threadIdx.x == 0) mbase[mesh_count] = carry;
}

// Bvh::refit (src/bvh.rs:176-205): leaf box = union of its primitives'
// boxes + 1e-4, interior box = union of the two children + 1e-4, computed
// bottom-up (the second child to arrive finishes the parent). Unions are
// exact, so the boxes equal the reference's reverse-order loop bit for bit.
// Unlike the reference, count/left_first are kept (see include/rtbvh.h).
__global__ void __launch_bounds__(kBlock)
    k_refit(DAabb* __restrict__ nodes, uint32_t node_count, const uint32_t* __restrict__ indices, uint32_t index_count,
            uint32_t prim_count,
            const DAabb* __restrict__ aabbs, const uint32_t* __restrict__ parent, uint32_t* __restrict__ arrive,
            uint32_t* __restrict__ status) {
  uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= node_count) return;
  DAabb nd = load_aabb_cg(nodes + c);
  if (nd.count < 0 && nd.left_first >= 0) return;  // interior: finished by a child walk
  DAabb box = nd;
  for (int a = 0; a < 3; ++a) { box.min[a] = 1e34f; box.max[a] = -1e34f; }
  if (nd.left_first >= 0) {
    for (int32_t i = 0; i < nd.count; ++i) {
      uint32_t slot = (uint32_t)nd.left_first + (uint32_t)i;
      if (slot >= index_count) { atomicOr(status, kStatusBadIndex); break; }
      uint32_t p = __ldg(indices + slot);
      if (p >= prim_count) { atomicOr(status, kStatusBadIndex); break; }
      DAabb b = load_aabb(aabbs + p);
      for (int a = 0; a < 3; ++a) { box.min[a] = rs_min(box.min[a], b.min[a]); box.max[a] = rs_max(box.max[a], b.max[a]); }
    }
    for (int a = 0; a < 3; ++a) { box.min[a] = box.min[a] - 0.0001f; box.max[a] = box.max[a] + 0.0001f; }
  }
  store_aabb(nodes + c, box);
  if (nd.left_first < 0) return;
  uint32_t x = c, w = __ldg(parent + c);
  for (uint32_t steps = 0; steps < node_count; ++steps) {
    if (w == kNone) break;
    const uint32_t p = parent_of(w);
    // topology words and the next parent are read while the arrival is under way
    const int32_t pc = __ldcg(&nodes[p].count), pl = __ldcg(&nodes[p].left_first);
    const uint32_t above = __ldg(parent + p);
    if (arrive_acq_rel(arrive + p) == 0u) break;
    const DAabb sib = load_aabb_cg(nodes + sibling_of(x, w));
    const bool right = (w & 1u) != 0u;  // the right child: the sibling's box comes first
    for (int a = 0; a < 3; ++a) {
      const float l0 = right ? sib.min[a] : box.min[a], r0 = right ? box.min[a] : sib.min[a];
      const float l1 = right ? sib.max[a] : box.max[a], r1 = right ? box.max[a] : sib.max[a];
      box.min[a] = rs_min(rs_min(1e34f, l0), r0) - 0.0001f;
      box.max[a] = rs_max(rs_max(-1e34f, l1), r1) + 0.0001f;
    }
    box.count = pc;
    box.left_first = pl;
    store_aabb(nodes + p, box);
    x = p;
    w = above;
  }
}

}  // namespace

ResultCode refit_bvh(DAabb* nodes, uint32_t node_count, const uint32_t* indices, uint32_t index_count,
                     uint32_t prim_count, const DAabb* aabbs, cudaStream_t s) {
  if (node_count == 0) return Ok;
  cudaError_t e;
  Scratch<uint32_t> parent, arrive, status;
  if ((e = parent.alloc(node_count, s)) || (e = arrive.alloc(node_count, s)) || (e = status.alloc(4, s)))
    return cuda_rc(e);
  if ((e = cudaMemsetAsync(parent.ptr, 0xff, (size_t)node_count * 4, s)) ||
      (e = cudaMemsetAsync(status.ptr, 0, 16, s)))
    return cuda_rc(e);
  const unsigned blocks = (node_count + kBlock - 1) / kBlock;
  k_parents<<<blocks, kBlock, 0, s>>>(nodes, node_count, parent.ptr, arrive.ptr, nullptr, nullptr, status.ptr);
  k_refit<<<blocks, kBlock, 0, s>>>(nodes, node_count, indices, index_count, prim_count, aabbs, parent.ptr,
                                    arrive.ptr, status.ptr);
  uint32_t st = 0;
  if ((e = cudaGetLastError()) || (e = cudaMemcpyAsync(&st, status.ptr, 4, cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s)))
    return cuda_rc(e);
  return st ? Error : Ok;
}

}  // namespace rtbvh

// ---------------------------------------------------------------- refit without allocation
// Variant of refit_bvh for callers that must not allocate device memory,
// for example a renderer that refits every frame inside a region where it
// is not allowed to call cudaMalloc (an allocation can synchronise the
// device and can fail mid-frame). Its scratch (parent pointers, arrival
// counters) lives in this file-scope array instead of being allocated per
// call; errors go to the Bvh's own status word. The array is reserved on a
// GPU when this module is first used there (with lazy module loading, at
// the latest on the first call) and stays reserved until the process exits.
namespace rtbvh {

namespace {

constexpr uint32_t kNoAllocHeadWords = 64;  // 256 bytes ahead of the arrays (unused), keeps them 256-byte aligned
static __device__ __align__(256) uint32_t g_refit_scratch[kNoAllocHeadWords + 2u * RTBVH_REFIT_NOALLOC_MAX_NODES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
uint32_t* g_noalloc_ptr[kMaxDevices] = {};

// Device address of g_refit_scratch on the current device, looked up once
// per device (with that device current) on its first use.
cudaError_t noalloc_scratch(uint32_t** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_refit_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = static_cast<uint32_t*>(p);
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace

ResultCode refit_bvh_noalloc(DAabb* nodes, uint32_t node_count, const uint32_t* indices, uint32_t index_count,
                             uint32_t prim_count, const DAabb* aabbs, uint32_t* status, cudaStream_t s) {
  if (node_count == 0) return Ok;
  if (node_count > RTBVH_REFIT_NOALLOC_MAX_NODES) return InvalidArgument;
  uint32_t* base = nullptr;
  cudaError_t e = noalloc_scratch(&base);
  if (e != cudaSuccess) return cuda_rc(e);
  uint32_t* parent = base + kNoAllocHeadWords;
  uint32_t* arrive = parent + RTBVH_REFIT_NOALLOC_MAX_NODES;
  // The array keeps the previous call's contents: reset what must start
  // clean (k_parents zeroes the arrival counters itself).
  if ((e = cudaMemsetAsync(parent, 0xff, (size_t)node_count * 4, s))) return cuda_rc(e);
  const unsigned blocks = (node_count + kBlock - 1) / kBlock;
  k_parents<<<blocks, kBlock, 0, s>>>(nodes, node_count, parent, arrive, nullptr, nullptr, status);
  k_refit<<<blocks, kBlock, 0, s>>>(nodes, node_count, indices, index_count, prim_count, aabbs, parent, arrive,
                                    status);
  return cuda_rc(cudaGetLastError());
}

}  // namespace rtbvh

// ---------------------------------------------------------------- compact quad nodes
namespace rtbvh {

namespace {

// One axis of a DQNode: grid start lo = the smallest bound of the four
// slots, step 2^k with 255 * 2^k covering the axis extent, lower bounds
// rounded down and upper bounds rounded up. The checks are exact: x - lo is
// split into hi + lo parts (two-sum, this file is compiled without
// contraction) and compared with q * 2^k, which is exact in float. False if a
// value is out of range or does not fit.
__device__ __forceinline__ void two_diff(float a, float b, float& hi, float& lo) {
  hi = a - b;
  const float bb = hi - a;
  lo = (a - (hi - bb)) + (-b - bb);
}

__device__ bool quantize_axis(const float* mn, const float* mx, float* lo_out, uint32_t* e_out, uint32_t* qlo,
                              uint32_t* qhi) {
  float lo = mn[0], hi = mn[0];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (!(fabsf(mn[i]) <= kQuantRange) || !(fabsf(mx[i]) <= kQuantRange)) return false;
    lo = fminf(lo, fminf(mn[i], mx[i]));
    hi = fmaxf(hi, fmaxf(mn[i], mx[i]));
  }
  int k = -126;
  const float ext = hi - lo;
  if (ext > 0.0f) {
    int ex;
    const float m = frexpf(ext / 255.0f, &ex);  // ext / 255 = m 2^ex, m in [0.5, 1)
    k = (m == 0.5f) ? ex - 1 : ex;
    if (k < -126) k = -126;
  }
  for (int attempt = 0; attempt < 3; ++attempt, ++k) {
    if (k > 127) return false;
    const float step = __uint_as_float((uint32_t)(k + 127) << 23);
    const float inv_step = (k <= 126) ? __uint_as_float((uint32_t)(127 - k) << 23) : 0.0f;
    if (k > 126 || k < -126) return false;
    uint32_t L = 0, H = 0;
    bool ok = true;
    for (int i = 0; i < 4 && ok; ++i) {
      float dh, dl;
      two_diff(mn[i], lo, dh, dl);  // mn - lo == dh + dl exactly
      float q = floorf(dh * inv_step);
      if (q < 0.0f) q = 0.0f;
      if (q > 255.0f) q = 255.0f;
      // need q * step <= dh + dl
      for (int g = 0; g < 4 && q > 0.0f; ++g) {
        const float v = q * step;
        if (v < dh || (v == dh && dl >= 0.0f)) break;
        q -= 1.0f;
      }
      {
        const float v = q * step;
        if (!(v < dh || (v == dh && dl >= 0.0f))) q = 0.0f;  // 0 is always below: lo is the minimum
      }
      const uint32_t ql = (uint32_t)q;
      two_diff(mx[i], lo, dh, dl);
      q = ceilf(dh * inv_step);
      if (q < 0.0f) q = 0.0f;
      // need q * step >= dh + dl
      for (int g = 0; g < 4; ++g) {
        const float v = q * step;
        if (v > dh || (v == dh && dl <= 0.0f)) break;
        q += 1.0f;
      }
      const float v = q * step;
      if (q > 255.0f || !(v > dh || (v == dh && dl <= 0.0f))) {
        ok = false;
      } else {
        L |= ql << (8 * i);
        H |= (uint32_t)q << (8 * i);
      }
    }
    if (ok) {
      *lo_out = lo;
      *e_out = (uint32_t)(k + 127);
      *qlo = L;
      *qhi = H;
      return true;
    }
  }
  return false;
}

__device__ void quantize_node(const DMNode& m, DQNode* out) {
  DQNode q;
  uint32_t ex = 0, ey = 0, ez = 0;
  bool ok = quantize_axis(m.min_x, m.max_x, &q.lo[0], &ex, &q.qx[0], &q.qx[1]) &&
            quantize_axis(m.min_y, m.max_y, &q.lo[1], &ey, &q.qy[0], &q.qy[1]) &&
            quantize_axis(m.min_z, m.max_z, &q.lo[2], &ez, &q.qz[0], &q.qz[1]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    q.children[k] = m.children[k];
    ok = ok && m.counts[k] >= -32768 && m.counts[k] <= 32767;
    q.counts[k] = (int16_t)m.counts[k];
  }
  if (!ok) {
    q.lo[0] = q.lo[1] = q.lo[2] = 0.0f;
    q.qx[0] = q.qx[1] = q.qy[0] = q.qy[1] = q.qz[0] = q.qz[1] = 0u;
    ex = ey = ez = 0;
  }
  bool in_range = true;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    in_range = in_range && fabsf(m.min_x[k]) <= kCompactRange && fabsf(m.max_x[k]) <= kCompactRange &&
               fabsf(m.min_y[k]) <= kCompactRange && fabsf(m.max_y[k]) <= kCompactRange &&
               fabsf(m.min_z[k]) <= kCompactRange && fabsf(m.max_z[k]) <= kCompactRange;
  const uint32_t flags = (ok ? 0u : kQFlagExact) | (in_range ? 0u : kQFlagOutOfRange);
  q.exps = ex | (ey << 8) | (ez << 16) | (flags << 24);
  const float4* src = reinterpret_cast<const float4*>(&q);
  float4* dst = reinterpret_cast<float4*>(out);
#pragma unroll
  for (int k = 0; k < 4; ++k) dst[k] = src[k];
}

}  // namespace

}  // namespace rtbvh

// ---------------------------------------------------------------- traversal tree (4-wide, tight boxes)
// A second 4-wide collapse of the BVH2 for the closest-hit traversal: each
// node takes the two children of its BVH2 node and keeps opening the
// interior child of largest half area until it has four slots (every slot
// keeps its own BVH2 box; the reference Mbvh instead gives a leaf slot its
// parent's box and opens strictly by depth). The tree is an internal
// acceleration structure: its boxes contain every triangle of their
// subtrees, so a traversal over it finds the same nearest hit.
//
// BVH2s whose boxes need not contain their triangles (a binned-SAH build;
// triangles attached after the build) get the same collapse over boxes
// recomputed from the triangles (build_mbvh with MbvhTriangles computes
// them), and their escaped triangles -- those that lie outside a box the
// reference's Mbvh tests on the way to them -- are flagged (mark_escapes).
// A ray that hits an escaped triangle (t below its current nearest) leaves
// the walk and is traced again over the exact Mbvh. For every other ray the
// nearest hit equals the reference's: (1) the walk's nearest triangle T is
// not escaped, so every box the reference tests on the way to T contains
// T, and the reference reaches T unless it already holds a nearer hit; (2)
// a triangle T' nearer than T that the reference reaches lies inside the
// walk's boxes, so the walk reaches and hits T' too -- it would have kept
// T' (not escaped) or handed the ray on.
namespace rtbvh {

namespace {

struct WideParams {
  const DAabb* nodes;  // boxes the tree is built over (BVH2, or its boxes from the triangles)
  uint32_t node_count;
  const uint32_t* parent;
  const uint64_t* cnt;  // nodes that are not counted are not below a root
  uint8_t* opened;      // per interior node: which of its descendants its traversal node would open
  uint32_t* index;      // per node: its traversal node, kNone for none
  uint32_t* roots;      // BVH2 node of every traversal node
  DMNode* wnodes;
  DQNode* wq;
  uint32_t capacity;
  uint32_t* walloc;     // next free traversal-node index (starts at 1; node 0 is BVH2 node 0's)
  uint32_t* status;
  // optional checks run before: nothing is built when check[0] != 0 (boxes
  // that do not nest, or duplicate leaf slots) or, with expect_seen != kNone,
  // when check[1] (primitives seen in leaves) differs from it
  uint32_t* check;
  uint32_t expect_seen;
  bool check_nested;
  // a forest: index of every mesh's root
  const uint32_t* prim_off;
  uint32_t mesh_count;
  uint32_t* qroot;
};

__device__ __forceinline__ bool interior(const DAabb& b) { return b.count < 0 && b.left_first >= 0; }

// A traversal node takes the two children of its BVH2 node as slots 0 and 1
// and opens up to two slots: each time the interior slot of largest half
// area (the first one of equals) is replaced by its left child, and the
// right child is appended. The code of a node: bits 0-1 the first opened slot
// + 1 (0: none), bits 2-3 the second opened slot + 1.
__device__ __forceinline__ int largest_interior(const DAabb* box, int ns) {
  int best = -1;
  float best_area = -1.0f;
  for (int i = 0; i < ns; ++i) {
    if (!interior(box[i])) continue;
    const float a = half_area(box[i].min[0], box[i].min[1], box[i].min[2], box[i].max[0], box[i].max[1],
                              box[i].max[2]);
    if (a > best_area) {
      best_area = a;
      best = i;
    }
  }
  return best;
}
// Whether code c opens its own child `side`.
__device__ __forceinline__ bool opens_child(uint32_t c, uint32_t side) {
  const uint32_t first = c & 3u, second = c >> 2;
  if (first == 0u) return false;
  return first == side + 1u || (second == side + 1u && first != side + 1u);
}
// Whether code c opens child `side2` of its own child `side`, which only the
// first opened child's children can be: its left one took its slot, its
// right one slot 2.
__device__ __forceinline__ bool opens_grandchild(uint32_t c, uint32_t side, uint32_t side2) {
  const uint32_t first = c & 3u, second = c >> 2;
  return first == side + 1u && second == (side2 ? 3u : first);
}

// The traversal tree without an order between levels. Which nodes a node
// would open if it had a traversal node of its own depends on the boxes
// below it alone, so every interior node computes its code at once
// (k_wide_open). A node then is the root of a traversal node (state R),
// opened by its parent (O1) or opened by its grandparent (O2), and its state
// follows from its parent's: R -> opens_child(parent) ? O1 : R,
// O1 -> opens_grandchild(grandparent) ? O2 : R, O2 -> R (a traversal node
// reaches three levels down at most). k_place composes these steps up to the
// first node whose step is the same from every state -- two or three levels
// on average -- and numbers the roots; k_wide_emit writes their nodes.
// What bounds it is the node reads, L2 for the most part; the level-by-level
// frontier it replaces spent a grid barrier per level: 200k sphere triangles
// 195 us, now k_wide_open 10, its part of k_place, k_wide_emit 15 us; 4M
// clustered 414 + 84 (compact nodes), now 93 and 167 us.
__global__ void __launch_bounds__(kBlock) k_wide_open(WideParams p) {
  const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= p.node_count) return;
  const bool below_root = counted(__ldg(p.cnt + c));
  if (!below_root && !p.check_nested) return;
  const DAabb cur = load_aabb(p.nodes + c);
  if (!interior(cur)) return;
  const uint32_t lf = (uint32_t)cur.left_first;
  if (lf + 1u >= p.node_count) {
    if (p.check_nested) atomicOr(p.check, 1u);
    return;
  }
  DAabb box[4];
  box[0] = load_aabb(p.nodes + lf);
  box[1] = load_aabb(p.nodes + lf + 1u);
  // Nesting check: every interior node's box contains both children's boxes.
  // The traversal tree finds the nearest hit only if the boxes it reads
  // contain their triangles, which holds for nested trees (leaf boxes are
  // always built from their primitives). A binned-SAH tree can violate it:
  // the reference sizes a left child's box from the bins before
  // best_splits[axis].count, a primitive count, instead of the split bin
  // (src/builders/binned_sah.rs), so the reference's own traversal can miss
  // hits there, and only its exact node order reproduces them.
  if (p.check_nested && !(box_contains(cur, box[0]) && box_contains(cur, box[1]))) atomicOr(p.check, 1u);
  if (!below_root) return;
  const int first = largest_interior(box, 2);
  int second = -1;
  if (first >= 0) {
    const uint32_t l2 = (uint32_t)box[first].left_first;
    if (l2 + 1u < p.node_count) {
      box[first] = load_aabb(p.nodes + l2);
      box[2] = load_aabb(p.nodes + l2 + 1u);
      second = largest_interior(box, 3);
    }
  }
  p.opened[c] = (uint8_t)((first + 1) | ((second + 1) << 2));
}

__device__ bool wide_checks_failed(const WideParams& p) {
  if (!p.check) return false;
  return __ldg(p.check) != 0u || (p.expect_seen != kNone && __ldg(p.check + 1) != p.expect_seen);
}

// Whether node x (below a root) is the root of a traversal node.
__device__ bool wide_root(const WideParams& p, uint32_t x) {
  // f: state of the current node -> x is in state R, one bit per state R, O1, O2
  uint32_t f = 1u;
  uint32_t cur = x;
  for (uint32_t k = 0; k < p.node_count; ++k) {
    const uint32_t w = __ldg(p.parent + cur);
    if (w == kNone) break;  // a tree's root: state R
    const uint32_t par = parent_of(w), side = w & 1u;
    const uint32_t gw = __ldg(p.parent + par);
    const bool a = opens_child(p.opened[par], side);
    const bool b = gw != kNone && opens_grandchild(p.opened[parent_of(gw)], gw & 1u, side);
    const uint32_t r = f & 1u, o1 = (f >> 1) & 1u, o2 = (f >> 2) & 1u;
    // state of the parent R, O1, O2 -> state of cur
    f = (a ? o1 : r) | ((b ? o2 : r) << 1) | (r << 2);
    if (f == 0u || f == 7u) break;
    cur = par;
  }
  return (f & 1u) != 0u;
}

// One thread per BVH2 node: places the interior ones (and the roots), lists
// the quad nodes among them by index and, with WIDE, numbers and lists the
// roots of traversal nodes.
template <bool TRIS, bool WIDE>
__global__ void __launch_bounds__(kBlock) k_place(CollapseParams p, WideParams q) {
  __shared__ uint32_t s_warp[kBlock / 32];
  __shared__ uint32_t s_base;
  const uint32_t x = blockIdx.x * kBlock + threadIdx.x;
  bool placed = x < p.node_count && counted(__ldg(p.cnt + x));
  if (placed) {
    const bool leaf = __ldg(&p.nodes[x].count) >= 0;
    placed = !leaf || (__ldg(p.parent + x) == kNone && ld_place(p.known + x).x != kNone);
  }
  if (placed) {
    const Place pl = find_place<TRIS>(p, x);
    placed = pl.ok;  // else not below a root
    if (placed) {
      st_place(p.known + x, make_uint2(pl.pos << 1 | pl.parity, pl.bad));
      if (pl.parity == 0u) {
        if (pl.pos < p.m_total) p.quads[pl.pos] = x;
        else atomicOr(p.status, kStatusBadIndex);
      }
    }
  }
  if (!WIDE) return;
  if (wide_checks_failed(q)) return;  // the same words for every block
  const bool root = placed && wide_root(q, x);
  // node 0 has traversal node 0 (the counter starts at 1)
  const uint32_t mine = root && x != 0u ? 1u : 0u;
  uint32_t total;
  const uint32_t incl = block_inclusive_scan<kBlock>(mine, s_warp, &total);
  if (threadIdx.x == 0) s_base = total ? atomicAdd(q.walloc, total) : 0u;
  __syncthreads();
  if (x >= p.node_count) return;
  const uint32_t wi = !root ? kNone : (mine ? s_base + incl - 1u : 0u);
  q.index[x] = wi;
  if (!root) return;
  if (wi < q.capacity) q.roots[wi] = x;
  else atomicOr(p.status, kStatusBadIndex);
}

__global__ void __launch_bounds__(kBlock) k_wide_emit(WideParams p) {
  if (wide_checks_failed(p)) return;
  const uint32_t wi = blockIdx.x * kBlock + threadIdx.x;
  for (uint32_t m = wi; m < p.mesh_count; m += gridDim.x * kBlock)
    p.qroot[m] = __ldg(p.index + 2u * __ldg(p.prim_off + m) - m);
  if (wi >= min(__ldg(p.walloc), p.capacity)) return;
  const uint32_t c = __ldg(p.roots + wi);
  if (c >= p.node_count) {  // not listed: only after another error
    atomicOr(p.status, kStatusBadIndex);
    return;
  }
  uint32_t slot[4];
  DAabb box[4];
  int ns = 0;
  const DAabb cur = load_aabb(p.nodes + c);
  if (!interior(cur)) {  // a root leaf
    slot[0] = c;
    box[0] = cur;
    ns = 1;
  } else {
    slot[0] = (uint32_t)cur.left_first;
    slot[1] = slot[0] + 1u;
    box[0] = load_aabb(p.nodes + slot[0]);
    box[1] = load_aabb(p.nodes + slot[1]);
    ns = 2;
    const uint32_t code = p.opened[c];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const int at = (int)((code >> (2 * o)) & 3u) - 1;
      if (at < 0) break;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (i != at) continue;
        const uint32_t lf = (uint32_t)box[i].left_first;
        if (lf + 1u >= p.node_count) {
          atomicOr(p.status, kStatusBadIndex);
          return;
        }
        slot[i] = lf;
        box[i] = load_aabb(p.nodes + lf);
        slot[2 + o] = lf + 1u;
        box[2 + o] = load_aabb(p.nodes + lf + 1u);
      }
      ++ns;
    }
  }
  DMNode m;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const DAabb& b = i < ns ? box[i] : box[0];
    m.min_x[i] = b.min[0]; m.min_y[i] = b.min[1]; m.min_z[i] = b.min[2];
    m.max_x[i] = b.max[0]; m.max_y[i] = b.max[1]; m.max_z[i] = b.max[2];
    m.children[i] = -1;
    m.counts[i] = -1;
    if (i < ns && !interior(b)) {
      m.children[i] = b.left_first;
      m.counts[i] = b.count;
    } else if (i < ns) {
      const uint32_t child = __ldg(p.index + slot[i]);
      if (child < p.capacity) m.children[i] = (int32_t)child;
      else atomicOr(p.status, kStatusBadIndex);
    }
  }
  store_node(p.wnodes + wi, m);
  quantize_node(m, p.wq + wi);
}

// The leaves of the object-split builders hold every index slot once and
// every primitive once, so their boxes cover whole primitives. Spatial-split
// trees (several fragments of a triangle, fragment boxes, unused slots) do
// not: any of those sets *bad.
__global__ void __launch_bounds__(kBlock) k_check_leaves(const DAabb* __restrict__ nodes, uint32_t node_count,
                                                         const uint32_t* __restrict__ indices, uint32_t index_count,
                                                         uint32_t* __restrict__ seen, uint32_t* __restrict__ total,
                                                         uint32_t* __restrict__ bad) {
  const uint32_t c = blockIdx.x * kBlock + threadIdx.x;
  if (c >= node_count) return;
  const DAabb n = load_aabb(nodes + c);
  if (n.count < 0 || n.left_first < 0) return;
  atomicAdd(total, (uint32_t)n.count);
  for (int32_t k = 0; k < n.count; ++k) {
    const uint32_t slot = (uint32_t)n.left_first + (uint32_t)k;
    if (slot >= index_count) {
      atomicOr(bad, 1u);
      return;
    }
    const uint32_t p = __ldg(indices + slot);
    if (p >= index_count || atomicAdd(seen + p, 1u) != 0u) {
      atomicOr(bad, 1u);
      return;
    }
  }
}

}  // namespace

// Scratch words per node of the collapse passes: parent, cnt (2), known (2),
// traversal index, the two lists of quad and traversal nodes (a
// forest of single leaves has as many as nodes), opened codes (a byte,
// rounded up).
size_t collapse_scratch_words(size_t node_count) { return 8 * node_count + (node_count + 3) / 4 + 8; }

namespace {

__global__ void k_set_word(uint32_t* p, uint32_t v) { *p = v; }

struct CollapseScratch {
  uint32_t *parent, *index, *quads, *roots;
  uint64_t* cnt;
  uint2* known;
  uint8_t* opened;
  // words holds collapse_scratch_words(node_count) words, 8-byte aligned
  CollapseScratch(uint32_t* words, size_t n) {
    cnt = reinterpret_cast<uint64_t*>(words);
    known = reinterpret_cast<uint2*>(cnt + n);
    parent = reinterpret_cast<uint32_t*>(known + n);
    index = parent + n;
    quads = index + n;
    roots = quads + n;
    opened = reinterpret_cast<uint8_t*>(roots + n);
  }
};

// Parents and counts (with `tri` also the boxes from the triangles).
cudaError_t launch_counts(const DAabb* nodes, uint32_t node_count, const CollapseScratch& w, const MbvhTriangles* tri,
                          uint32_t* status, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(w.parent, 0xff, (size_t)node_count * 4, s))) return e;
  const unsigned blocks = (node_count + kBlock - 1) / kBlock;
  k_parents<<<blocks, kBlock, 0, s>>>(nodes, node_count, w.parent, nullptr, w.cnt, w.known, status);
  const unsigned count_blocks = (node_count + kCountBlock - 1) / kCountBlock;
  if (tri)
    k_counts_bottom_up<true><<<count_blocks, kCountBlock, 0, s>>>(nodes, node_count, w.parent, w.cnt, *tri, status);
  else
    k_counts_bottom_up<false><<<count_blocks, kCountBlock, 0, s>>>(nodes, node_count, w.parent, w.cnt, MbvhTriangles(),
                                                        status);
  return cudaGetLastError();
}

// The quad nodes and, with q, the traversal nodes.
cudaError_t launch_nodes(const CollapseParams& p, bool tris, const WideParams* q, cudaStream_t s) {
  const unsigned blocks = (p.node_count + kBlock - 1) / kBlock, quad_blocks = (p.m_total + kBlock - 1) / kBlock;
  if (q) k_wide_open<<<blocks, kBlock, 0, s>>>(*q);
  auto place = tris ? (q ? k_place<true, true> : k_place<true, false>)
                    : (q ? k_place<false, true> : k_place<false, false>);
  place<<<blocks, kBlock, 0, s>>>(p, q ? *q : WideParams());
  auto quads = tris ? k_quads<true> : k_quads<false>;
  quads<<<quad_blocks, kBlock, 0, s>>>(p);
  if (q) k_wide_emit<<<(q->capacity + kBlock - 1) / kBlock, kBlock, 0, s>>>(*q);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_collapse_forest(const DAabb* nodes, uint32_t node_count, const uint32_t* prim_off,
                                   uint32_t mesh_count, uint32_t total_prims, uint32_t* scratch, uint32_t* mbase,
                                   DMNode* mnodes, DMNode* wnodes, DQNode* wq, uint32_t* qroot, uint32_t* walloc,
                                   uint32_t* status, cudaStream_t s) {
  if (node_count == 0 || mesh_count == 0) return cudaSuccess;
  cudaError_t e;
  const CollapseScratch w(scratch, node_count);
  if ((e = launch_counts(nodes, node_count, w, nullptr, status, s))) return e;
  k_seg_mbase<<<1, 1024, 0, s>>>(nodes, w.cnt, prim_off, mesh_count, w.known, mbase);
  CollapseParams p = {};
  p.nodes = nodes;
  p.node_count = node_count;
  p.parent = w.parent;
  p.cnt = w.cnt;
  p.known = w.known;
  p.quads = w.quads;
  p.mnodes = mnodes;
  p.m_total = total_prims;  // a mesh of n > 1 primitives has at most n - 1 interior nodes
  p.m_count = mbase + mesh_count;
  p.forest = true;
  p.status = status;
  if (!wnodes) return launch_nodes(p, false, nullptr, s);
  WideParams q = {};
  q.nodes = nodes;
  q.node_count = node_count;
  q.parent = w.parent;
  q.cnt = w.cnt;
  q.opened = w.opened;
  q.index = w.index;
  q.roots = w.roots;
  q.wnodes = wnodes;
  q.wq = wq;
  q.capacity = total_prims;
  q.walloc = walloc;
  q.status = status;
  q.expect_seen = kNone;
  q.prim_off = prim_off;
  q.mesh_count = mesh_count;
  q.qroot = qroot;
  k_set_word<<<1, 1, 0, s>>>(walloc, 1u);
  return launch_nodes(p, false, &q, s);
}

ResultCode build_mbvh(const DAabb* nodes, uint32_t node_count, cudaStream_t s, const MbvhRequest& req, MbvhOutput* out) {
  *out = MbvhOutput();
  if (node_count == 0) return Ok;  // Mbvh::default()
  const MbvhTriangles* tri = req.tri;
  if (tri && (!tri->indices || !tri->vertices || !tri->tris || !tri->tb)) return Error;
  // The node counts stay on the device until the end; arrays are sized by
  // their bounds: quad nodes are interior BVH2 nodes, at most
  // (node_count - 1) / 2 of a binary tree, or the root leaf; the same holds
  // for traversal nodes.
  const uint32_t m_cap = (node_count + 1u) / 2u;
  const bool check_nested = req.wide && !tri;
  const uint32_t* check_indices = req.wide ? req.check_indices : nullptr;
  cudaError_t e;
  Scratch<uint32_t> seen;
  ScratchPack scratch;
  // result words: 0 status, 1 check (not nested, duplicate leaf slots), 2
  // primitives in leaves, 3 escaped triangles, 4 quad nodes, 5 traversal nodes,
  // 6 the root's box misses triangles
  uint32_t *words, *res;
  scratch.add(&words, collapse_scratch_words(node_count));
  scratch.add(&res, 8);
  if ((e = scratch.alloc(s))) return cuda_rc(e);
  auto drop = [&](ResultCode rc) {
    pool_free(out->mnodes, s);
    pool_free(out->tboxes, s);
    pool_free(out->wnodes, s);
    pool_free(out->wq, s);
    *out = MbvhOutput();
    return rc;
  };
  if ((e = device_alloc(&out->mnodes, m_cap, s))) return drop(cuda_rc(e));
  if (tri && (e = device_alloc(&out->tboxes, m_cap, s))) return drop(cuda_rc(e));
  if (req.wide && ((e = device_alloc(&out->wnodes, m_cap, s)) || (e = device_alloc(&out->wq, m_cap, s))))
    return drop(cuda_rc(e));
  if ((e = cudaMemsetAsync(res, 0, 32, s))) return drop(cuda_rc(e));
  const CollapseScratch w(words, node_count);
  if ((e = launch_counts(nodes, node_count, w, tri, res, s))) return drop(cuda_rc(e));
  const unsigned blocks = (node_count + kBlock - 1) / kBlock;
  k_root_place<<<1, 32, 0, s>>>(w.cnt, nodes, w.known, m_cap, res + 4, res + 5, res + 6, res);
  CollapseParams p = {};
  p.nodes = nodes;
  p.node_count = node_count;
  p.parent = w.parent;
  p.cnt = w.cnt;
  p.known = w.known;
  p.quads = w.quads;
  p.mnodes = out->mnodes;
  p.m_total = m_cap;
  p.m_count = res + 4;
  p.status = res;
  if (tri) p.tri = *tri;
  p.escaped = res + 3;
  p.tboxes = out->tboxes;
  if (!req.wide) {
    if ((e = launch_nodes(p, tri != nullptr, nullptr, s))) return drop(cuda_rc(e));
  } else {
    if (check_indices) {
      if ((e = seen.alloc(req.index_count, s)) || (e = cudaMemsetAsync(seen.ptr, 0, (size_t)req.index_count * 4, s)))
        return drop(cuda_rc(e));
      k_check_leaves<<<blocks, kBlock, 0, s>>>(nodes, node_count, check_indices, req.index_count, seen.ptr,
                                               res + 2, res + 1);
    }
    WideParams q = {};
    q.nodes = tri ? tri->tb : nodes;
    q.node_count = node_count;
    q.parent = w.parent;
    q.cnt = w.cnt;
    q.opened = w.opened;
    q.index = w.index;
    q.roots = w.roots;
    q.wnodes = out->wnodes;
    q.wq = out->wq;
    q.capacity = m_cap;
    q.walloc = res + 5;
    q.status = res;
    q.check = res + 1;
    q.check_nested = check_nested;
    q.expect_seen = check_indices ? req.index_count : kNone;
    if ((e = launch_nodes(p, tri != nullptr, &q, s))) return drop(cuda_rc(e));
  }
  uint32_t h[7];
  if ((e = cudaGetLastError()) || (e = cudaMemcpyAsync(h, res, sizeof(h), cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s)))
    return drop(cuda_rc(e));
  if (h[0] != 0) return drop((h[0] & kStatusTimeout) ? Timeout : Error);
  out->mcount = h[4];
  out->escaped = h[3];
  out->bad_root = h[6] != 0;
  if (req.wide && (h[1] || (check_indices && h[2] != req.index_count))) {
    // no traversal tree: closest hit reads the exact nodes
    pool_free(out->wnodes, s);
    pool_free(out->wq, s);
    out->wnodes = nullptr;
    out->wq = nullptr;
  } else if (req.wide) {
    out->wcount = h[5];
    if (out->wcount == 0 || out->wcount > m_cap) return drop(Error);
  }
  return Ok;
}

}  // namespace rtbvh
