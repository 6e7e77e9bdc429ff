// Single-ray traversal with the fused triangle test, one ray per thread.
//
// trace_mbvh follows MbvhIndexIterator::next (src/iter_indices.rs:264-313)
// step for step: the quad node's hit mask and slot order come from the
// 4-wide slab test (src/mbvh_node.rs:176-240) evaluated with the ray's
// current t when the node is entered; slots are visited far to near
// (ids[3..0]); a leaf slot's primitives are tested at once, an interior slot
// is pushed. The triangle test is SpatialTriangle::intersect
// (src/builders/spatial_sah.rs:132-163). With the same arithmetic (no FMA,
// IEEE division, SSE min/max rules) the hits, their order of discovery and
// the node/triangle counts equal the reference's.
//
// trace_bvh follows BvhIndexIterator::next (src/iter_indices.rs:66-107) with
// the sign-indexed slab test (src/aabb.rs:145-181) and sort_nodes
// (src/bvh_node.rs:150-177).
//
// Kernels are persistent. The stack lives in local memory with a hard bound;
// a ray that would exceed it stops, reports prim -2 and sets
// kStatusStackOverflow. A quad node (one 128-byte line) is read with four
// 256-bit loads (each lane reads its own node, so the load count per node
// sets the L1 wavefronts). Leaf triangles are 64 bytes ({v0, prim}, {e1},
// {e2}, pad): two 256-bit loads.
//
// Closest hit without statistics reads the 64-byte compact copies of the
// quad nodes (DQNode, two 256-bit loads) when they exist: the boxes contain
// the exact ones, so the nearest triangle and its t/u/v are unchanged, and
// only the winner among triangles hit at exactly the same t can differ from
// the reference's visit order. (All of this for hits that lie in their
// triangles' boxes: nearly in a triangle's plane the test's t can be noise, see
// kTestError, and which such hits a walk finds depends on its boxes and order.)
// This halves the node bytes and the L1 fill
// traffic. Any hit, statistics and rays with a zero, non-finite or huge
// component use the exact nodes.
#include <cstdlib>

#include "lib_internal.h"

namespace rtbvh {

namespace {

constexpr int kBlock = 128;
constexpr int kStack = 64;

struct RayState {
  float ox, oy, oz, dx, dy, dz, ix, iy, iz;
  float t;
  int32_t sx, sy, sz;
};

__device__ __forceinline__ RayState load_ray(const float* rays, size_t r, const float* t_max) {
  const float2* p = reinterpret_cast<const float2*>(rays + 6 * r);
  float2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  RayState s;
  s.ox = a.x; s.oy = a.y; s.oz = b.x;
  s.dx = b.y; s.dy = c.x; s.dz = c.y;
  s.ix = 1.0f / s.dx; s.iy = 1.0f / s.dy; s.iz = 1.0f / s.dz;
  s.sx = s.dx < 0.0f; s.sy = s.dy < 0.0f; s.sz = s.dz < 0.0f;
  s.t = t_max ? __ldg(t_max + r) : 1e34f;
  return s;
}

// One 256-bit read-only load (sm_100+): 8 floats from a 32-byte aligned address.
__device__ __forceinline__ void ld8(const float* p, float (&v)[8]) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "l"(p));
}

// SpatialTriangle::intersect with a leaf-ordered triangle {v0,prim},{e1},{e2}.
__device__ __forceinline__ bool mt_test(const float4* tri, RayState& r, float& hu, float& hv, int32_t& prim) {
  float t0[8], t1[8];
  ld8(reinterpret_cast<const float*>(tri), t0);
  ld8(reinterpret_cast<const float*>(tri) + 8, t1);
  const float4 a = make_float4(t0[0], t0[1], t0[2], t0[3]), b = make_float4(t0[4], t0[5], t0[6], t0[7]);
  const float4 c = make_float4(t1[0], t1[1], t1[2], t1[3]);
  const float e1x = b.x, e1y = b.y, e1z = b.z;
  const float e2x = c.x, e2y = c.y, e2z = c.z;
  // h = d x e2
  const float hx = r.dy * e2z - e2y * r.dz;
  const float hy = r.dz * e2x - e2z * r.dx;
  const float hz = r.dx * e2y - e2x * r.dy;
  const float det = ((e1x * hx) + (e1y * hy)) + (e1z * hz);
  if (det > -1e-5f && det < 1e-5f) return false;
  const float f = 1.0f / det;
  const float sx = r.ox - a.x, sy = r.oy - a.y, sz = r.oz - a.z;
  const float u = f * (((sx * hx) + (sy * hy)) + (sz * hz));
  if (!(u >= 0.0f && u <= 1.0f)) return false;
  // q = s x e1
  const float qx = sy * e1z - e1y * sz;
  const float qy = sz * e1x - e1z * sx;
  const float qz = sx * e1y - e1x * sy;
  const float v = f * (((r.dx * qx) + (r.dy * qy)) + (r.dz * qz));
  if (v < 0.0f || (u + v) > 1.0f) return false;
  const float t = f * (((e2x * qx) + (e2y * qy)) + (e2z * qz));
  if (t > 1e-4f && t < r.t) {
    r.t = t;
    hu = u;
    hv = v;
    prim = __float_as_int(a.w);
    return true;
  }
  return false;
}

// Margins on the slab values of the three axes for walks that skip slots (see
// kTestError), infinite where none may be skipped.
struct SlabMargin {
  float x, y, z;
  __device__ __forceinline__ void set(const RayState& r, float distance) {
    x = distance * fabsf(r.ix);
    y = distance * fabsf(r.iy);
    z = distance * fabsf(r.iz);
  }
  __device__ __forceinline__ void set_none() { x = y = z = __int_as_float(0x7f800000); }
  // Whether a box with these exit values reaches the origin.
  __device__ __forceinline__ bool reaches(float tx, float ty, float tz) const { return tx >= -x && ty >= -y && tz >= -z; }
};

// MbvhNode::intersect: mask bit i set when slot i is hit; ids packed as
// 2-bit fields, ascending by t_min after the 5-compare network.
//
// FAST: for a ray whose origin, direction and inverse direction are all
// finite, no slab value can be NaN ((m - o) * inv with finite factors), and
// then the SSE select rule (a < b ? a : b) and the native min/max instruction
// return the same value; at most the sign of a zero differs, which no later
// comparison can see. So the fast form takes every decision the exact form
// takes. Rays with a zero or non-finite component use the exact form.
//
// BEHIND (FAST only): slots that lie behind the origin by the margin are left
// out of the mask.
template <bool FAST, bool BEHIND = false>
__device__ __forceinline__ void quad_intersect(const DMNode* node, const RayState& r, uint32_t& mask, uint32_t& ids,
                                               int4& children, int4& counts, const SlabMargin& behind = {}) {
  const float* q = reinterpret_cast<const float*>(node);
  float vx[8], vy[8], vz[8], vc[8];
  ld8(q, vx);
  ld8(q + 8, vy);
  ld8(q + 16, vz);
  ld8(q + 24, vc);
  const float4 mnx = make_float4(vx[0], vx[1], vx[2], vx[3]), mxx = make_float4(vx[4], vx[5], vx[6], vx[7]);
  const float4 mny = make_float4(vy[0], vy[1], vy[2], vy[3]), mxy = make_float4(vy[4], vy[5], vy[6], vy[7]);
  const float4 mnz = make_float4(vz[0], vz[1], vz[2], vz[3]), mxz = make_float4(vz[4], vz[5], vz[6], vz[7]);
  const float4 ch = make_float4(vc[0], vc[1], vc[2], vc[3]), ct = make_float4(vc[4], vc[5], vc[6], vc[7]);
  children = make_int4(__float_as_int(ch.x), __float_as_int(ch.y), __float_as_int(ch.z), __float_as_int(ch.w));
  counts = make_int4(__float_as_int(ct.x), __float_as_int(ct.y), __float_as_int(ct.z), __float_as_int(ct.w));
  float tmin[4];
  uint32_t m = 0;
  const float a_mnx[4] = {mnx.x, mnx.y, mnx.z, mnx.w}, a_mxx[4] = {mxx.x, mxx.y, mxx.z, mxx.w};
  const float a_mny[4] = {mny.x, mny.y, mny.z, mny.w}, a_mxy[4] = {mxy.x, mxy.y, mxy.z, mxy.w};
  const float a_mnz[4] = {mnz.x, mnz.y, mnz.z, mnz.w}, a_mxz[4] = {mxz.x, mxz.y, mxz.z, mxz.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float tx0 = (a_mnx[i] - r.ox) * r.ix, tx1 = (a_mxx[i] - r.ox) * r.ix;
    const float ty0 = (a_mny[i] - r.oy) * r.iy, ty1 = (a_mxy[i] - r.oy) * r.iy;
    const float tz0 = (a_mnz[i] - r.oz) * r.iz, tz1 = (a_mxz[i] - r.oz) * r.iz;
    float tn, tx;
    bool reaches = true;
    if (FAST) {
      const float txx = fmaxf(tx0, tx1), tyx = fmaxf(ty0, ty1), tzx = fmaxf(tz0, tz1);
      tn = fmaxf(fminf(tx0, tx1), fmaxf(fminf(ty0, ty1), fminf(tz0, tz1)));
      tx = fminf(txx, fminf(tyx, tzx));
      if (BEHIND) reaches = behind.reaches(txx, tyx, tzx);
    } else {
      const float txn = sse_min(tx0, tx1), txx = sse_max(tx0, tx1);
      const float tyn = sse_min(ty0, ty1), tyx = sse_max(ty0, ty1);
      const float tzn = sse_min(tz0, tz1), tzx = sse_max(tz0, tz1);
      tn = sse_max(txn, sse_max(tyn, tzn));
      tx = sse_min(txx, sse_min(tyx, tzx));
    }
    tmin[i] = tn;
    if ((tx >= tn) && (tn < r.t) && reaches) m |= 1u << i;
  }
  uint32_t i0 = 0, i1 = 1, i2 = 2, i3 = 3;
  float t0 = tmin[0], t1 = tmin[1], t2 = tmin[2], t3 = tmin[3], tt;
  uint32_t ti;
  if (t0 > t1) { tt = t0; t0 = t1; t1 = tt; ti = i0; i0 = i1; i1 = ti; }
  if (t2 > t3) { tt = t2; t2 = t3; t3 = tt; ti = i2; i2 = i3; i3 = ti; }
  if (t0 > t2) { tt = t0; t0 = t2; t2 = tt; ti = i0; i0 = i2; i2 = ti; }
  if (t1 > t3) { tt = t1; t1 = t3; t3 = tt; ti = i1; i1 = i3; i3 = ti; }
  if (t2 > t3) { ti = i2; i2 = i3; i3 = ti; }
  mask = m;
  ids = i0 | (i1 << 2) | (i2 << 4) | (i3 << 6);
}

// Slot bound q of a DQNode axis word as the float q * 2^-133 (exact): the
// byte is moved to bits 16-23 with zeros around it, which is a denormal below
// 128 and the smallest normal binade above, the same line q * 2^-133. One
// instruction, where an offset in the mantissa needed a subtraction as well.
// The factor goes into the step (kStepBias), so that the slab products come
// out times kKeyScale, a power of two, and round as before down to keys of
// 2^-54; nearer the origin they are denormal and lose bits, which can reorder
// visits at such distances (the boxes' margin is 1e-4). The walk is
// bound by its issue rate; 24 subtractions fewer of about 250 instructions per
// node, with counts decoded only for tested leaves and the pushes counted at
// once: 16.8M incoherent rays over 1M triangles 16.07 -> 14.13 ms, 4.2M camera
// rays over 200k triangles 1.65 -> 1.42 ms.
__device__ __forceinline__ float qbyte(uint32_t w, uint32_t i) {
  return __int_as_float((int)__byte_perm(w, 0u, 0x4044u | (i << 8)));
}
// Steps are at most 2 (bounds within kCompactRange), inverse directions below
// 2^60: (step * 2^61) * inv stays below 2^122, and (step * 2^61) * inv * q *
// 2^-133 is the slab product times 2^-72.
constexpr uint32_t kStepBias = 61u << 23;
constexpr float kKeyScale = 2.117582368135750836e-22f;  // 2^-72

__device__ __forceinline__ bool finite_ray(const RayState& r) {
  return isfinite(r.ox) && isfinite(r.oy) && isfinite(r.oz) && isfinite(r.dx) && isfinite(r.dy) && isfinite(r.dz) &&
         isfinite(r.ix) && isfinite(r.iy) && isfinite(r.iz);
}

__device__ __forceinline__ int sel4(const int4& v, uint32_t i) {
  return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

// Per-lane ray refill shared by the persistent MBVH kernels: a lane whose ray
// has finished takes the next ray from a warp-local pool (refilled `batch`
// rays at a time from the global counter), so the warp's lanes stay busy
// instead of idling until the warp's slowest ray ends.
// Default rays per pool refill (TraceArgs::ray_batch). Small batches keep the
// end of a launch short (the last warps hold few rays); measured on one GB300
// against 128: the 1M incoherent scene +0.9 %, the 6,400-triangle sphere's
// camera +20 %, the 200k-triangle camera -4 % time (64, 16: less on one or
// the other; 256, 512: slower everywhere).
constexpr uint32_t kPoolBatch = 32;

struct WarpPool {
  uint32_t next = 0, end = 0;  // warp-uniform (ray counts < 2^32 - 2^25)
  bool exhausted = false;      // warp-uniform
  // Calls start(k) on every lane that is not active, for the next unclaimed
  // ray positions k; start decides whether the lane becomes active. Idle lanes
  // wait until there are IDLE of them (unless no lane is active), so that the
  // ray set-up, which only the refilled lanes execute, runs for that many
  // lanes at a time. Any hit, 4.2M shadow rays over 1M triangles with 2, 4, 6,
  // 8 lanes: 3,620, 3,596, 3,598, 3,660 us; closest hits over the exact nodes,
  // 1M rays over 1M triangles with 2 and 4: 4,294, 4,343.
  template <int IDLE, class Start>
  __device__ __forceinline__ void refill(bool active, uint32_t batch, uint32_t ray_count, unsigned int* work,
                                         Start&& start) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t need = __ballot_sync(0xffffffffu, !active);
    if (!need || (__popc(need) < IDLE && need != 0xffffffffu)) return;
    // first from what is left in the pool ...
    const uint32_t avail = end - next;
    if (avail) {
      const uint32_t rank = __popc(need & lt_mask);
      const bool mine = (need >> lane) & 1u;
      if (mine && rank < avail) start(next + rank);
      const uint32_t c = __popc(need);
      next += c < avail ? c : avail;
      need = __ballot_sync(0xffffffffu, mine && rank >= avail);
    }
    // ... then from a fresh batch of the global counter
    if (need) {
      unsigned int base = 0;
      if (lane == 0) base = atomicAdd(work, batch);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= ray_count) {
        exhausted = true;
      } else {
        next = base;
        end = (ray_count - base > batch) ? base + batch : ray_count;
        const uint32_t avail2 = end - next;
        const bool mine = (need >> lane) & 1u;
        const uint32_t rank = __popc(need & lt_mask);
        if (mine && rank < avail2) start(next + rank);
        const uint32_t c = __popc(need);
        next += c < avail2 ? c : avail2;
      }
    }
  }
};

// Mesh of ray r in a forest: m with seg_ray_off[m] <= r < seg_ray_off[m + 1].
__device__ __forceinline__ uint32_t ray_mesh(const TraceArgs& a, uint32_t r) {
  uint32_t lo = 0, hi = a.seg_count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(a.seg_ray_off + mid) <= r) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Whether a ray with the bound t may have a hit in a box with these entry and
// exit values of the axes.
template <bool ANY_HIT>
__device__ __forceinline__ bool enters(float nx, float ny, float nz, float fx, float fy, float fz, float t,
                                       const SlabMargin& m) {
  if (!ANY_HIT) {
    const float tn = fmaxf(nx, fmaxf(ny, nz)), tx = fminf(fx, fminf(fy, fz));
    return tx >= tn && tx >= 0.0f && tn < t;
  }
  const float tn = fmaxf(nx - m.x, fmaxf(ny - m.y, nz - m.z)), tx = fminf(fx + m.x, fminf(fy + m.y, fz + m.z));
  return tx >= tn && tx >= 0.0f && tn < t;
}

// Hit mask of a quad node's subtree boxes (DTBox): slot i is set when the
// ray can enter its box at some t in [0, r.t). Finite rays within the
// compact walk's range only (the rounding argument of kCompactRange: a box
// that holds a triangle hit at t > 1e-4 passes), any hit with a margin
// (kTestError).
template <bool ANY_HIT>
__device__ __forceinline__ uint32_t subtree_mask(const DTBox* box, const RayState& r, const SlabMargin& margin) {
  const float* q = reinterpret_cast<const float*>(box);
  float vx[8], vy[8], vz[8];
  ld8(q, vx);
  ld8(q + 8, vy);
  ld8(q + 16, vz);
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float tx0 = (vx[i] - r.ox) * r.ix, tx1 = (vx[4 + i] - r.ox) * r.ix;
    const float ty0 = (vy[i] - r.oy) * r.iy, ty1 = (vy[4 + i] - r.oy) * r.iy;
    const float tz0 = (vz[i] - r.oz) * r.iz, tz1 = (vz[4 + i] - r.oz) * r.iz;
    if (enters<ANY_HIT>(fminf(tx0, tx1), fminf(ty0, ty1), fminf(tz0, tz1), fmaxf(tx0, tx1), fmaxf(ty0, ty1),
                        fmaxf(tz0, tz1), r.t, margin))
      m |= 1u << i;
  }
  return m;
}

// ------------------------------------------------------------------ four lanes per ray
// Few rays leave most of the GPU idle and the launch as long as its longest
// walk: then four neighbouring lanes take a ray together, one slot of a node
// each, which shortens a node visit to the test of one slot and a few
// shuffles. The visits, their order and the result are those of the walks
// with a lane per ray: the slots go through the same sorting network, lane by
// lane, and where the leaves of one node are tested side by side, a hit counts
// if no leaf before it in the walk's order has a nearer one.
struct FourLanes {
  uint32_t first;  // lane 0 of the four
  uint32_t l;      // this lane of the four
  __device__ __forceinline__ FourLanes() : first(threadIdx.x & 28u), l(threadIdx.x & 3u) {}
  template <class T>
  __device__ __forceinline__ T from(T v, uint32_t k) const {
    return __shfl_sync(0xffffffffu, v, (int)(first + k));
  }
  __device__ __forceinline__ uint32_t ballot(bool b) const {
    return (__ballot_sync(0xffffffffu, b) >> first) & 15u;
  }
};

// Warps that `rays` rays are spread over, at most eight to a warp: about
// kFewWarpsPerScheduler for each of an SM's four schedulers as long as there
// are rays for that many. Ray i goes to warp i % warps.
constexpr uint32_t kFewWarpsPerScheduler = 3;
// Launches of at most so many rays take four lanes per ray. Closest hit, one
// lane against four, in us: 4,096 rays 102 / 76 (6,400-triangle sphere, SAH),
// 246 / 226 (200k soup, LOCB), 301 / 224 (300k clustered, SAH); 16,384: 111 /
// 98, 264 / 255, 315 / 245; 32,768: 102 / 78, 273 / 298, 317 / 261. Any hit
// (300k clustered): 4,096 rays 194 / 132, 65,536: 281 / 235, 131,072: 301 /
// 319. Rays handed on by the compact walk come from binned-SAH trees; up to
// kFewDeferred of them take four lanes. So do more, up to kFewDeferredMost,
// where they are a small part of their launch: that part is the rays with the
// longest walks, so the longest chain counts and not the throughput. One lane
// against four, in us: 4M rays of which 68k are handed on 5,607 / 4,580 (2M
// clustered), 4.2M of which 83k 1,882 / 1,677 (200k sphere), 16M of which 270k
// 14,770 / 13,970; 1/4 to 1/32 of the launch as the line: all the same. Where
// whole launches are handed on (scenes beyond the compact walk's range) one
// lane per ray is the better from about 131k rays, and 1.4 times at 262k.
constexpr uint32_t kFewClosest = 20480, kFewAny = 65536;
constexpr uint32_t kFewDeferred = 32768, kFewDeferredMost = 524288, kFewDeferredPart = 16;
__device__ __host__ __forceinline__ uint32_t few_warps(uint32_t rays, uint32_t sms) {
  const uint32_t spread = sms * 4u * kFewWarpsPerScheduler;
  const uint32_t least = (rays + 7u) / 8u;
  return least > spread ? least : (rays < spread ? rays : spread);
}

// Best of the four lanes' hits of one node: t is every lane's nearest t (the
// entry t where it has none). HIGH_FIRST: the walk tests the leaves of higher
// lanes first, else those of lower lanes. Returns the lane of the first
// nearest hit, -1 for none below `entry`, and the nearest t of the lanes
// before this one.
template <bool HIGH_FIRST>
__device__ __forceinline__ int first_nearest(const FourLanes& q, float t, float entry, float& best, float& before) {
  const float t0 = q.from(t, 0), t1 = q.from(t, 1), t2 = q.from(t, 2), t3 = q.from(t, 3);
  best = fminf(fminf(t0, t1), fminf(t2, t3));
  before = entry;
  if (HIGH_FIRST) {
    if (q.l < 3u) before = fminf(before, t3);
    if (q.l < 2u) before = fminf(before, t2);
    if (q.l < 1u) before = fminf(before, t1);
  } else {
    if (q.l > 0u) before = fminf(before, t0);
    if (q.l > 1u) before = fminf(before, t1);
    if (q.l > 2u) before = fminf(before, t2);
  }
  if (!(best < entry)) return -1;
  if (HIGH_FIRST) return t3 == best ? 3 : (t2 == best ? 2 : (t1 == best ? 1 : 0));
  return t0 == best ? 0 : (t1 == best ? 1 : (t2 == best ? 2 : 3));
}

constexpr int kCullNone = 0, kCullSubtree = 1, kCullBehind = 2;  // see k_trace_mbvh

// How far the float triangle test may be off, for any-hit walks that skip
// slots. In exact arithmetic, with s = o - v0 and an accepted (t, u, v),
//   det (o + t d - v0 - u e1 - v e2) = dDet s + dT d - dU e1 - dV e2
// where dDet .. dV are the rounding errors of the determinant and of the
// numerators of t, u and v. The roundings of mt_test (2^-24 each) add up to at
// most 5.9, 7.3, 6.9 and 7.3 times 2^-24 |e1| |e2| |d| |s| for the four terms,
// and an accepted |det| is at least 1e-5: the point o + t d lies within
//   0.17 |e1| |e2| |d| |s|  (27.4 * 2^-24 / 1e-5)
// of the triangle, and 1.6e-6 |s| more for the roundings of t d and of the edges
// themselves (no edge is longer than 2 |s| with s the farthest corner). A ray
// nearly in a triangle's plane gets that far: t is noise there. Over the
// each direction component that distance, less what the boxes' own growth
// takes up, is a margin on the axis's slab values. |s| is at most the distance
// of the root box's farthest corner, |e1| |e2| the largest of the tree's
// triangles but for the few large ones of TriEdges. Those are tested with the
// ray first: one that such a triangle accepts outside its own box skips nothing,
// and scenes with more of them skip nothing at all.
// 4.2M shadow rays over 1M clustered triangles, us: 3,790; 3,600 without the
// margins (and with other hits on such rays); 4,300 with the largest margin of
// the axes for all three, which needs one comparison instead of three, where
// directions with a small component skip little; 4,610 with each slot's
// squared diagonal for |e1| |e2|; 5,490 with each slot's farthest corner for |s|.
constexpr float kTestError = 0.17f, kTestErrorRest = 1.6e-6f;
constexpr float kBoxSlack = 5e-5f;  // of the 1e-4 that boxes are grown by, what the slab test's rounding leaves

// Whether one of the large triangles accepts this ray outside its own box.
__device__ __forceinline__ bool large_noise(const TraceArgs& a, uint32_t large, const RayState& ray,
                                            const SlabMargin& margin) {
#pragma unroll 1
  for (uint32_t k = 0; k < large; ++k) {
    const uint32_t slot = __ldg(a.edges->slot + k);
    if (slot >= a.prim_count) return true;
    const float4* tri = a.tris + kTriFloat4 * (size_t)slot;
    RayState r = ray;
    float u, v;
    int32_t p;
    if (!mt_test(tri, r, u, v, p)) continue;
    // slab values of its box, which lies inside every box on the way to it
    const float4 v0 = __ldg(tri), e1 = __ldg(tri + 1), e2 = __ldg(tri + 2);
    float n[3], f[3];
    auto slab = [&](int k, float x, float ax, float bx, float o, float i) {
      const float t0 = (fminf(x, fminf(x + ax, x + bx)) - o) * i, t1 = (fmaxf(x, fmaxf(x + ax, x + bx)) - o) * i;
      n[k] = fminf(t0, t1);
      f[k] = fmaxf(t0, t1);
    };
    slab(0, v0.x, e1.x, e2.x, ray.ox, ray.ix);
    slab(1, v0.y, e1.y, e2.y, ray.oy, ray.iy);
    slab(2, v0.z, e1.z, e2.z, ray.oz, ray.iz);
    if (!enters<true>(n[0], n[1], n[2], f[0], f[1], f[2], ray.t, margin)) return true;
  }
  return false;
}

// Whether slots may be skipped for this ray, and (any hit) the margin, infinite
// where they may not.
template <bool ANY_HIT, int CULL>
__device__ __forceinline__ bool cull_ray(const TraceArgs& a, const RayState& ray, SlabMargin& margin) {
  margin.set_none();
  const DAabb root = load_aabb(a.nodes);
  // |x| <= bound is false for NaN and infinities
  bool cull = fabsf(ray.ox) <= kCompactRange && fabsf(ray.oy) <= kCompactRange && fabsf(ray.oz) <= kCompactRange &&
              fabsf(ray.dx) <= 3.0e38f && fabsf(ray.dy) <= 3.0e38f && fabsf(ray.dz) <= 3.0e38f &&
              fabsf(ray.ix) <= kQuantRange && fabsf(ray.iy) <= kQuantRange && fabsf(ray.iz) <= kQuantRange;
  if (CULL == kCullSubtree) {
    // Only rays that start inside the scene's root box: boxes behind
    // them are most of what the cull saves; for rays from outside the
    // extra box loads cost more than they save
    cull = cull && ray.ox >= root.min[0] && ray.oy >= root.min[1] && ray.oz >= root.min[2] &&
           ray.ox <= root.max[0] && ray.oy <= root.max[1] && ray.oz <= root.max[2];
  } else {
    // the margin argument needs the boxes within the range too
    for (int k = 0; k < 3; ++k) cull = cull && root.min[k] >= -kCompactRange && root.max[k] <= kCompactRange;
    // rays that enter the scene from outside have nothing behind them
    const float tn = fmaxf(fminf((root.min[0] - ray.ox) * ray.ix, (root.max[0] - ray.ox) * ray.ix),
                           fmaxf(fminf((root.min[1] - ray.oy) * ray.iy, (root.max[1] - ray.oy) * ray.iy),
                                 fminf((root.min[2] - ray.oz) * ray.iz, (root.max[2] - ray.oz) * ray.iz)));
    cull = cull && tn < 0.0f;
  }
  if (!ANY_HIT || !cull) return cull;
  const uint32_t large = __ldg(&a.edges->large);
  const float x = fmaxf(fabsf(ray.ox - root.min[0]), fabsf(ray.ox - root.max[0]));
  const float y = fmaxf(fabsf(ray.oy - root.min[1]), fabsf(ray.oy - root.max[1]));
  const float z = fmaxf(fabsf(ray.oz - root.min[2]), fabsf(ray.oz - root.max[2]));
  const float far = sqrtf(x * x + y * y + z * z);
  const float len = sqrtf(ray.dx * ray.dx + ray.dy * ray.dy + ray.dz * ray.dz);
  const float off = far * (kTestError * __ldg(&a.edges->product) * len + kTestErrorRest);
  if (!(off <= 1.0e18f) || large > kLargeTriangles) return false;
  margin.set(ray, fmaxf(0.0f, off - kBoxSlack));
  if (large && large_noise(a, large, ray, margin)) {
    margin.set_none();
    return false;
  }
  return true;
}

// Start of ray r's walk over the quad nodes: the root (of its mesh); false:
// no nodes, a miss.
__device__ __forceinline__ bool mbvh_root(const TraceArgs& a, uint32_t r, int32_t& root) {
  root = 0;
  if (a.node_count == 0) return false;
  if (a.seg_count) {
    const uint32_t m = ray_mesh(a, r);
    root = (int32_t)__ldg(a.seg_root + m);
    if ((uint32_t)root == __ldg(a.seg_root + m + 1)) return false;
  }
  return true;
}

// One lane's slot of a quad node.
struct LaneQuad {
  float x0, x1, y0, y1, z0, z1;
  int32_t child, count;
  __device__ __forceinline__ void load(const DMNode* node, uint32_t l) {
    const float* n = reinterpret_cast<const float*>(node) + l;
    x0 = __ldg(n);
    x1 = __ldg(n + 4);
    y0 = __ldg(n + 8);
    y1 = __ldg(n + 12);
    z0 = __ldg(n + 16);
    z1 = __ldg(n + 20);
    child = __float_as_int(__ldg(n + 24));
    count = __float_as_int(__ldg(n + 28));
  }
};

// k_trace_mbvh's walk, four lanes per ray, for ray_count rays. The next node
// is popped and asked for before the leaves are tested. The four lanes share
// one stack in `shared`, or, without it, each keeps the whole of it: as a
// branch of k_trace_mbvh the shared stacks took L1 from the other branch (1M
// rays beyond the compact walk's range over a 200k soup 3,770 -> 3,830 us).
template <bool ANY_HIT, int CULL, bool SHARED>
__device__ void walk_mbvh4(const TraceArgs& a, uint32_t ray_count, uint32_t warps, int32_t* shared) {
  const FourLanes q;
  int32_t own[SHARED ? 1 : kStack];
  int32_t* const stack = SHARED ? shared : own;
  const uint32_t warp = blockIdx.x * (kBlock / 32u) + (threadIdx.x >> 5);
  RayState ray;
  float hu = 0.0f, hv = 0.0f;
  int32_t prim = -1, current = -1;  // the node whose slots are in `slot`
  int sp = -1;
  bool active = false, fast = true, cull = false;
  SlabMargin margin;
  margin.set_none();
  uint32_t r = 0;
  LaneQuad slot;
  auto fetch = [&]() {
    if ((uint32_t)current >= a.node_count) {
      if (q.l == 0u) atomicOr(a.status, kStatusBadIndex);
      active = false;
    } else {
      slot.load(a.mnodes + current, q.l);
    }
  };
  for (size_t i = warp < warps ? warp + (size_t)warps * (q.first >> 2) : ray_count;;) {
    if (!active && i < ray_count) {
      r = a.order ? __ldg(a.order + i) : (uint32_t)i;
      i += 8u * (size_t)warps;
      ray = load_ray(a.rays, r, a.t_max);
      fast = finite_ray(ray);
      if (CULL != kCullNone && a.node_count > 0) cull = cull_ray<ANY_HIT, CULL>(a, ray, margin);
      hu = hv = 0.0f;
      prim = -1;
      sp = -1;
      active = mbvh_root(a, r, current);
      if (active) fetch();
      else if (q.l == 0u) a.hits[r] = make_float4(ray.t, 0.0f, 0.0f, __int_as_float(-1));
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (!__any_sync(0xffffffffu, i < ray_count)) break;
      continue;
    }
    // own slot, then the network of quad_intersect over the four lanes
    float t = __int_as_float(0x7f800000);
    int32_t child = -1, count = -1;
    bool hit = false;
    if (active) {
      const float tx0 = (slot.x0 - ray.ox) * ray.ix, tx1 = (slot.x1 - ray.ox) * ray.ix;
      const float ty0 = (slot.y0 - ray.oy) * ray.iy, ty1 = (slot.y1 - ray.oy) * ray.iy;
      const float tz0 = (slot.z0 - ray.oz) * ray.iz, tz1 = (slot.z1 - ray.oz) * ray.iz;
      child = slot.child;
      count = slot.count;
      float tx;
      bool reaches = true;
      if (fast) {
        const float txx = fmaxf(tx0, tx1), tyx = fmaxf(ty0, ty1), tzx = fmaxf(tz0, tz1);
        t = fmaxf(fminf(tx0, tx1), fmaxf(fminf(ty0, ty1), fminf(tz0, tz1)));
        tx = fminf(txx, fminf(tyx, tzx));
        if (CULL == kCullBehind) reaches = margin.reaches(txx, tyx, tzx);
      } else {
        t = sse_max(sse_min(tx0, tx1), sse_max(sse_min(ty0, ty1), sse_min(tz0, tz1)));
        tx = sse_min(sse_max(tx0, tx1), sse_min(sse_max(ty0, ty1), sse_max(tz0, tz1)));
      }
      hit = (tx >= t) && (t < ray.t) && reaches;
      if (CULL == kCullSubtree && cull && hit) {
        const float* b = reinterpret_cast<const float*>(a.tboxes + current) + q.l;
        const float bx0 = (__ldg(b) - ray.ox) * ray.ix, bx1 = (__ldg(b + 4) - ray.ox) * ray.ix;
        const float by0 = (__ldg(b + 8) - ray.oy) * ray.iy, by1 = (__ldg(b + 12) - ray.oy) * ray.iy;
        const float bz0 = (__ldg(b + 16) - ray.oz) * ray.iz, bz1 = (__ldg(b + 20) - ray.oz) * ray.iz;
        hit = enters<ANY_HIT>(fminf(bx0, bx1), fminf(by0, by1), fminf(bz0, bz1), fmaxf(bx0, bx1), fmaxf(by0, by1),
                              fmaxf(bz0, bz1), ray.t, margin);
      }
    }
    const uint32_t hits = q.ballot(hit);
    uint32_t id = q.l;
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      const float ot = __shfl_xor_sync(0xffffffffu, t, o);
      const uint32_t oid = __shfl_xor_sync(0xffffffffu, id, o);
      const bool low = (q.l & (uint32_t)o) == 0u;
      if (low ? t > ot : ot > t) {
        t = ot;
        id = oid;
      }
    }
    {
      const float ot = __shfl_xor_sync(0xffffffffu, t, 1);
      const uint32_t oid = __shfl_xor_sync(0xffffffffu, id, 1);
      if (q.l >= 2u && (q.l == 2u ? t > ot : ot > t)) id = oid;
    }
    // the slot at this lane's place; places are visited from 3 down to 0
    child = q.from(child, id);
    count = q.from(count, id);
    hit = (hits >> id) & 1u;
    const bool inner = hit && count <= -1 && child > -1;
    bool leaf = hit && count > -1;
    const uint32_t inners = q.ballot(inner);
    const int n = __popc(inners);
    const int32_t nearest = q.from(child, inners ? (uint32_t)__ffs(inners) - 1u : 0u);
    bool done = false, push = false, overflow = false;
    int32_t next = -1;
    if (n > 0) {
      next = nearest;
      if (sp + n - 1 >= kStack) {
        // the walk ends at the slot whose push does not fit: the first interior
        // one needs none, then kStack - 1 - sp fit
        uint32_t rest = inners;
        for (int fit = kStack - sp; fit > 0; --fit) rest &= ~(0x80000000u >> __clz(rest));
        leaf = leaf && q.l > 31u - (uint32_t)__clz(rest);
        done = overflow = true;
      } else {
        push = true;
      }
    }
    // farther slots below nearer ones
    if (SHARED) {
      if (push) {
        if (inner && (inners & ((1u << q.l) - 1u))) stack[sp + 1 + __popc(inners >> (q.l + 1u))] = child;
        sp += n - 1;
      }
      __syncwarp();
    } else {
#pragma unroll
      for (uint32_t k = 3; k > 0; --k) {
        const int32_t c = q.from(child, k);
        if (push && ((inners >> k) & 1u) && (inners & ((1u << k) - 1u))) stack[++sp] = c;
      }
    }
    if (active && !done) {
      current = next;
      if (next < 0 && sp >= 0) current = stack[sp--];
      if (current >= 0) fetch();
    }
    if (__any_sync(0xffffffffu, leaf)) {
      const float entry = ray.t;
      float u = hu, v = hv;
      int32_t p = prim;
      bool bad = false, found = false;
      if (leaf) {
        bad = child < 0 || (uint32_t)child + (uint32_t)count > a.prim_count;
        if (bad) atomicOr(a.status, kStatusBadIndex);
        for (int32_t j = 0; !bad && j < count; ++j) {
          if (mt_test(a.tris + kTriFloat4 * (size_t)(child + j), ray, u, v, p)) {
            found = true;
            if (ANY_HIT) break;
          }
        }
      }
      const uint32_t founds = q.ballot(found);
      if (q.ballot(bad)) {
        done = true;
        overflow = false;
      }
      float best, before;
      int w = first_nearest<true>(q, ray.t, entry, best, before);
      if (ANY_HIT) w = founds ? 31 - __clz(founds) : -1;  // the first leaf in the walk's order
      const uint32_t src = w < 0 ? q.l : (uint32_t)w;
      const float wt = q.from(ray.t, src), wu = q.from(u, src), wv = q.from(v, src);
      const int32_t wp = q.from(p, src);
      ray.t = entry;
      if (w >= 0) {
        ray.t = wt;
        hu = wu;
        hv = wv;
        prim = wp;
        if (ANY_HIT) {
          done = true;
          overflow = false;
        }
      }
    }
    if (overflow) {
      if (q.l == 0u) atomicOr(a.status, kStatusStackOverflow);
      prim = -2;
    }
    if (active && (done || current < 0)) {
      if (q.l == 0u) a.hits[r] = make_float4(ray.t, hu, hv, __int_as_float(prim));
      active = false;
    }
  }
}

// Few rays over the exact quad nodes.
template <bool ANY_HIT, int CULL>
__global__ void __launch_bounds__(kBlock) k_trace_mbvh4(TraceArgs a, uint32_t warps) {
  __shared__ int32_t s_stack[kBlock / 4][kStack];
  walk_mbvh4<ANY_HIT, CULL, true>(a, (uint32_t)a.ray_count, warps, s_stack[threadIdx.x >> 2]);
}

// Persistent MBVH traversal over the exact quad nodes with per-lane ray
// refill. Each loop iteration visits one quad node per lane; a ray's
// node/triangle order is the reference's. With ray_count_dev the number of
// rays is read from the device (the rays the compact kernel deferred).
//
// CULL: slots that cannot hold a hit are skipped; the reference would walk
// their subtrees and accept nothing in them, so t and the order of all later
// tests are unchanged and the hit is the reference's bit for bit (the node
// counts are not, so STATS never culls).
//  kCullSubtree (binned-SAH trees with a.tboxes): slots whose subtree box
//   (from the triangles) the ray cannot enter below its current t.
//  kCullBehind (any hit over a tree whose slot boxes contain their triangles
//   grown by 1e-4, a.quads_cover): slots behind the origin, by the exit
//   values the slab test has anyway. What bounds such a walk is the
//   number of boxes visited: the slab test has no lower bound on t, so a
//   shadow ray that leaves a surface walks the whole scene behind it too.
//   4.2M shadow rays over 1M clustered triangles: 9,155 us without the skip,
//   3,790 with it. Rays that enter the scene from outside have nothing
//   behind them: warps with only such rays leave the comparisons out (1M
//   rays into a 200k soup, us: 2,230 with them, 2,165 without; 2,100 without
//   any of this).
//  Any hit leaves both a margin for the rounding of the triangle test
//   (kTestError), so that the hit is the reference's on grazing rays too.
//   Closest hit leaves none, like the compact walk: a hit that the triangle
//   test reports by rounding, outside the triangle's boxes, can be missed there.
// FEW: a launch whose ray count is read from the device walks with four lanes
// per ray when that is at most kFewDeferred. The launch bounds keep that
// branch from taking registers from the other one: 8 blocks per SM, 7 with
// subtree boxes (8 spill there). Without them 68 and 78 registers, and launches
// handed on whole were 5 to 10 % slower (1M rays, 1M clustered triangles:
// 6,190 us for 5,770; 200k sphere, SAH: 4,260 for 3,880).
// Any hit, leaves in one loop and 8 blocks per SM asked for (64 registers; 7
// take 72 and 4,040 us, 9 spill: 5,080 without the margins): those shadow rays
// 3,790 us, over the binned-SAH tree 4,240 (9,145 without the skip).
template <bool ANY_HIT, bool STATS, int CULL = kCullNone, bool FEW = false>
__global__ void __launch_bounds__(kBlock, (ANY_HIT && !STATS) ? 8 : FEW ? (CULL ? 7 : 8) : 0)
    k_trace_mbvh(TraceArgs a, unsigned int* work) {
  RayState ray;
  float hu = 0.0f, hv = 0.0f;
  int32_t prim = -1;
  uint32_t visits = 0, tests = 0, max_depth = 0;
  // The node to visit next is kept in `next` instead of on the stack: the
  // last child a node pushes is always the next one popped, so holding it in
  // a register saves one store and one load per visited node. The logical
  // stack is stack[0..sp] followed by `next` (when next >= 0).
  int32_t stack[kStack];
  int sp = -1;
  int32_t next = -1;
  uint32_t r = 0;
  bool active = false, fast = true, cull = false;
  bool culls = false;  // warp-uniform: some ray of the warp skips slots
  SlabMargin margin;
  margin.set_none();
  WarpPool pool;
  uint32_t batch = a.ray_batch ? a.ray_batch : kPoolBatch;
  const uint32_t ray_count = a.ray_count_dev ? *a.ray_count_dev : (uint32_t)a.ray_count;
  if (FEW) {
    if (ray_count <= kFewDeferred ||
        (ray_count <= kFewDeferredMost && ray_count <= a.ray_count / kFewDeferredPart)) {
      const uint32_t launched = gridDim.x * (kBlock / 32u), wanted = few_warps(ray_count, a.sms);
      walk_mbvh4<ANY_HIT, CULL, false>(a, ray_count, wanted < launched ? wanted : launched, nullptr);
      return;
    }
  }
  if (a.ray_count_dev) {
    // few rays (deferred by the compact walk): spread them over all warps,
    // down to one ray per refill, so that their walks run side by side
    const uint32_t warps = gridDim.x * (kBlock / 32u), even = ray_count / warps;
    batch = even < 1u ? 1u : (even < batch ? even : batch);
  }
  auto start_ray = [&](uint32_t rr) {
    r = a.order ? __ldg(a.order + rr) : rr;
    ray = load_ray(a.rays, r, a.t_max);
    fast = finite_ray(ray);
    if (CULL != kCullNone && a.node_count > 0) cull = cull_ray<ANY_HIT, CULL>(a, ray, margin);
    hu = hv = 0.0f;
    prim = -1;
    visits = tests = max_depth = 0;
    if (a.node_count == 0) {
      a.hits[r] = make_float4(ray.t, 0.0f, 0.0f, __int_as_float(-1));
      if (STATS) {
        a.stats[3 * (size_t)r + 0] = 0;
        a.stats[3 * (size_t)r + 1] = 0;
        a.stats[3 * (size_t)r + 2] = 0;
      }
    } else {
      sp = -1;
      next = 0;
      active = true;
      if (a.seg_count) {
        const uint32_t m = ray_mesh(a, r);
        const uint32_t root = __ldg(a.seg_root + m);
        if (root == __ldg(a.seg_root + m + 1)) {
          active = false;
          a.hits[r] = make_float4(ray.t, 0.0f, 0.0f, __int_as_float(-1));
          if (STATS) {
            a.stats[3 * (size_t)r + 0] = 0;
            a.stats[3 * (size_t)r + 1] = 0;
            a.stats[3 * (size_t)r + 2] = 0;
          }
        }
        next = (int32_t)root;
      }
    }
  };
  for (;;) {
    if (!pool.exhausted) {
      pool.refill<ANY_HIT ? 4 : 2>(active, batch, ray_count, work, start_ray);
      if (CULL == kCullBehind) culls = __any_sync(0xffffffffu, active && cull);
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (pool.exhausted) break;
      continue;
    }
    if (!active) continue;
    // ---- one quad node
    const int32_t current = next >= 0 ? next : stack[sp--];
    next = -1;
    if ((uint32_t)current >= a.node_count) {
      atomicOr(a.status, kStatusBadIndex);
      active = false;
      continue;
    }
    uint32_t mask, ids;
    int4 children, counts;
    bool done = false;
    if (CULL == kCullBehind && fast && culls)
      quad_intersect<true, true>(a.mnodes + current, ray, mask, ids, children, counts, margin);
    else if (fast) quad_intersect<true>(a.mnodes + current, ray, mask, ids, children, counts);
    else quad_intersect<false>(a.mnodes + current, ray, mask, ids, children, counts);
    if (CULL == kCullSubtree && cull) mask &= subtree_mask<ANY_HIT>(a.tboxes + current, ray, margin);
    if (STATS) ++visits;
    if (ANY_HIT && !STATS && mask == 0u) {
      // nothing to do: most visits of rays that miss (16.8M rays ending short
      // of the scene 318 -> 265 us)
    } else if (ANY_HIT && !STATS && sp + 4 < kStack) {
      // An accepted triangle ends the walk whatever the node pushed, so the
      // pushes go first and the leaves' triangles follow in one loop, in their
      // order; slot by slot, every slot was a loop of its own for the few
      // lanes with a leaf there.
      uint32_t leaves = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t id = (ids >> (2 * (3 - i))) & 3u;
        const int32_t count = sel4(counts, id), lf = sel4(children, id);
        if ((mask >> id) & 1u) {
          if (count > -1) {
            leaves |= 1u << i;
          } else if (lf > -1) {
            if (next >= 0) stack[++sp] = next;
            next = lf;
          }
        }
      }
      int32_t j = 0;
#pragma unroll 1
      while (leaves) {
        const uint32_t id = (ids >> (2 * (4 - __ffs(leaves)))) & 3u;
        const int32_t count = sel4(counts, id), lf = sel4(children, id);
        if (lf < 0 || (uint32_t)lf + (uint32_t)count > a.prim_count) {
          atomicOr(a.status, kStatusBadIndex);
          done = true;
          break;
        }
        if (j < count && mt_test(a.tris + kTriFloat4 * (size_t)(lf + j), ray, hu, hv, prim)) {
          done = true;
          break;
        }
        if (++j >= count) {
          leaves &= leaves - 1u;
          j = 0;
        }
      }
    } else
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      const uint32_t id = (ids >> (2 * (3 - i))) & 3u;
      if (!((mask >> id) & 1u)) continue;
      const int32_t count = sel4(counts, id);
      const int32_t lf = sel4(children, id);
      if (count > -1) {
        if (lf < 0 || (uint32_t)lf + (uint32_t)count > a.prim_count) {
          atomicOr(a.status, kStatusBadIndex);
          done = true;
          break;
        }
        bool hit_stop = false;
        for (int32_t j = 0; j < count; ++j) {
          if (STATS) ++tests;
          if (mt_test(a.tris + kTriFloat4 * (size_t)(lf + j), ray, hu, hv, prim) && ANY_HIT) {
            hit_stop = true;
            break;
          }
        }
        if (hit_stop) {
          done = true;
          break;
        }
      } else if (lf > -1) {
        if (next >= 0) {
          if (sp + 1 >= kStack) {
            atomicOr(a.status, kStatusStackOverflow);
            prim = -2;
            done = true;
            break;
          }
          stack[++sp] = next;
        }
        next = lf;
        if (STATS && (uint32_t)(sp + 2) > max_depth) max_depth = (uint32_t)(sp + 2);
      }
    }
    if (done || (next < 0 && sp < 0)) {
      a.hits[r] = make_float4(ray.t, hu, hv, __int_as_float(prim));
      if (STATS) {
        a.stats[3 * (size_t)r + 0] = visits;
        a.stats[3 * (size_t)r + 1] = tests;
        a.stats[3 * (size_t)r + 2] = max_depth;
      }
      active = false;
    }
  }
}

// Interior slots of a traversal-tree node in near-to-far order. key[i] is
// the entry t of the i-th nearest interior slot the ray hits; other slots
// (missed, empty, or leaves) get +inf and sort last. Each key's child
// travels with it through the sorting network, so the caller reads children
// by position without run-time indexing. A hit slot's key is finite: it is
// below the ray's t (no NaN arises on the compact path's finite rays).
__device__ __forceinline__ void sort_slots(float (&key)[4], int32_t (&ch)[4]) {
  auto cswap = [&](int a, int b) {
    const bool s = key[b] < key[a];
    const float ka = key[a], kb = key[b];
    const int32_t ca = ch[a], cb = ch[b];
    key[a] = s ? kb : ka;
    key[b] = s ? ka : kb;
    ch[a] = s ? cb : ca;
    ch[b] = s ? ca : cb;
  };
  cswap(0, 1);
  cswap(2, 3);
  cswap(0, 2);
  cswap(1, 3);
  cswap(1, 2);
}

// Key of slot i (interior slots only) and its bit in the leaf mask.
//
// A slot whose box lies wholly behind the origin (exit t below 0) is
// skipped as well, which the reference's test does not do: every box of a
// traversal tree contains its triangles grown by 1e-4, so a triangle hit at
// t > 1e-4 (the triangle test's lower bound) lies inside its boxes with that
// margin, and the box's computed exit t stays above 0 (the slab rounding is
// below the margin, see kCompactRange). The cull removes no box that holds
// such a hit (one that the test reports by rounding, outside its triangle's
// box, can go with it, see kTestError); it saves the walks of rays that start
// inside the scene (secondary rays) through the boxes behind them.
__device__ __forceinline__ void slot_key(float tn, float tx, float t, int32_t child, bool inner, int i, float& key,
                                         uint32_t& leaves) {
  const bool hit = tx >= tn && tx >= 0.0f && tn < t && child >= 0;
  key = (hit && inner) ? tn : __int_as_float(0x7f800000);
  leaves |= (hit && !inner) ? 1u << i : 0u;
}


// q0 * a + b and q1 * a + b in one instruction (two fmas, rounded as fmaf).
__device__ __forceinline__ void fma2(float q0, float q1, float a, float b, float& r0, float& r1) {
  asm("{\n\t.reg .b64 q, f, c, r;\n\t"
      "mov.b64 q, {%2, %3};\n\tmov.b64 f, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
      "fma.rn.f32x2 r, q, f, c;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r0), "=f"(r1)
      : "f"(q0), "f"(q1), "f"(a), "f"(b));
}

// The slab test of quad_intersect<true> on a compact node: the plane of step
// q is at lo + q * step, so its ray parameter is q * (step * inv) +
// (lo - o) * inv (one fma). With a negative inverse direction the upper
// plane is the near one; the fma is monotonic in q, so selecting the planes
// by sign equals min/max of the two. Outputs: the sorted interior keys and
// children, the hit leaf slots as a mask over the node's own slot order, and
// the node's children and counts in that order.
__device__ __forceinline__ void slot_keys_q(const float (&h0)[8], const float (&h1)[8], const RayState& r,
                                            float (&key)[4], int32_t (&ich)[4], uint32_t& leaves,
                                            int32_t (&ch)[4], uint32_t (&ct)[2]) {
  const uint32_t exps = __float_as_uint(h0[3]);
  const float sx = __uint_as_float(((exps & 0xffu) << 23) + kStepBias);
  const float sy = __uint_as_float(((exps >> 8 & 0xffu) << 23) + kStepBias);
  const float sz = __uint_as_float(((exps >> 16 & 0xffu) << 23) + kStepBias);
  const float ax = sx * r.ix, bx = (h0[0] - r.ox) * r.ix * kKeyScale;
  const float ay = sy * r.iy, by = (h0[1] - r.oy) * r.iy * kKeyScale;
  const float az = sz * r.iz, bz = (h0[2] - r.oz) * r.iz * kKeyScale;
  const float t = r.t * kKeyScale;
  const uint32_t xl = __float_as_uint(h0[4]), xh = __float_as_uint(h0[5]);
  const uint32_t yl = __float_as_uint(h0[6]), yh = __float_as_uint(h0[7]);
  const uint32_t zl = __float_as_uint(h1[0]), zh = __float_as_uint(h1[1]);
  const uint32_t xn = r.ix < 0.0f ? xh : xl, xf = r.ix < 0.0f ? xl : xh;
  const uint32_t yn = r.iy < 0.0f ? yh : yl, yf = r.iy < 0.0f ? yl : yh;
  const uint32_t zn = r.iz < 0.0f ? zh : zl, zf = r.iz < 0.0f ? zl : zh;
  ct[0] = __float_as_uint(h1[6]);
  ct[1] = __float_as_uint(h1[7]);
  ch[0] = __float_as_int(h1[2]);
  ch[1] = __float_as_int(h1[3]);
  ch[2] = __float_as_int(h1[4]);
  ch[3] = __float_as_int(h1[5]);
  // two slots per instruction: 12 issue slots fewer per node, 2 % on every
  // kind of rays
  float nx[4], ny[4], nz[4], fx[4], fy[4], fz[4];
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    fma2(qbyte(xn, i), qbyte(xn, i + 1), ax, bx, nx[i], nx[i + 1]);
    fma2(qbyte(yn, i), qbyte(yn, i + 1), ay, by, ny[i], ny[i + 1]);
    fma2(qbyte(zn, i), qbyte(zn, i + 1), az, bz, nz[i], nz[i + 1]);
    fma2(qbyte(xf, i), qbyte(xf, i + 1), ax, bx, fx[i], fx[i + 1]);
    fma2(qbyte(yf, i), qbyte(yf, i + 1), ay, by, fy[i], fy[i + 1]);
    fma2(qbyte(zf, i), qbyte(zf, i + 1), az, bz, fz[i], fz[i + 1]);
  }
  leaves = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float tn = fmaxf(nx[i], fmaxf(ny[i], nz[i])), tx = fminf(fx[i], fminf(fy[i], fz[i]));
    const bool inner = (ct[i >> 1] & (0x8000u << (16 * (i & 1)))) != 0u;
    slot_key(tn, tx, t, ch[i], inner, i, key[i], leaves);
    ich[i] = ch[i];
  }
  sort_slots(key, ich);
}

// The same from a node's exact (128-byte) copy, for compact nodes whose
// bounds did not fit the grid; FAST arithmetic (finite rays only). `large`: a
// leaf of more primitives than 15 bits count.
__device__ __forceinline__ void slot_keys_exact(const DMNode* node, const RayState& r, float (&key)[4],
                                                int32_t (&ich)[4], uint32_t& leaves, int32_t (&ch)[4],
                                                uint32_t (&ct)[2], bool& large) {
  const float* q = reinterpret_cast<const float*>(node);
  float vx[8], vy[8], vz[8], vc[8];
  ld8(q, vx);
  ld8(q + 8, vy);
  ld8(q + 16, vz);
  ld8(q + 24, vc);
  leaves = 0;
  // counts of 16 bits, as in the compact node
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int32_t c0 = __float_as_int(vc[4 + 2 * k]), c1 = __float_as_int(vc[5 + 2 * k]);
    large = large || c0 > 32767 || c1 > 32767;
    ct[k] = ((uint32_t)c0 & 0xffffu) | ((uint32_t)c1 << 16);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ch[i] = __float_as_int(vc[i]);
    const float tx0 = (vx[i] - r.ox) * r.ix, tx1 = (vx[4 + i] - r.ox) * r.ix;
    const float ty0 = (vy[i] - r.oy) * r.iy, ty1 = (vy[4 + i] - r.oy) * r.iy;
    const float tz0 = (vz[i] - r.oz) * r.iz, tz1 = (vz[4 + i] - r.oz) * r.iz;
    const float tn = fmaxf(fminf(tx0, tx1), fmaxf(fminf(ty0, ty1), fminf(tz0, tz1)));
    const float tx = fminf(fmaxf(tx0, tx1), fminf(fmaxf(ty0, ty1), fmaxf(tz0, tz1)));
    slot_key(tn, tx, r.t, ch[i], __float_as_int(vc[4 + i]) < 0, i, key[i], leaves);
    ich[i] = ch[i];
  }
  sort_slots(key, ich);
}

// Whether the compact walk takes this ray (|x| <= bound is false for NaN and
// infinities).
__device__ __forceinline__ bool compact_ray(const RayState& ray) {
  return fabsf(ray.ox) <= kCompactRange && fabsf(ray.oy) <= kCompactRange && fabsf(ray.oz) <= kCompactRange &&
         fabsf(ray.dx) <= 3.0e38f && fabsf(ray.dy) <= 3.0e38f && fabsf(ray.dz) <= 3.0e38f &&
         fabsf(ray.ix) <= kQuantRange && fabsf(ray.iy) <= kQuantRange && fabsf(ray.iz) <= kQuantRange;
}
// Start of ray r's walk over the traversal tree (of its mesh); false: no
// nodes, a miss.
__device__ __forceinline__ bool compact_root(const TraceArgs& a, uint32_t r, int32_t& root) {
  root = 0;
  if (a.node_count == 0) return false;
  if (a.seg_count) {
    const uint32_t m = ray_mesh(a, r);
    if (__ldg(a.seg_root + m) == __ldg(a.seg_root + m + 1)) return false;
    root = (int32_t)__ldg(a.seg_qroot + m);
  }
  return true;
}

// Closest hit over the compact (64-byte) nodes of the traversal tree, with
// the leaf tests taken out of the slot loop. A loop iteration has a node
// phase -- each lane with no untested leaf visits its next node, pushes the
// node's hit interior slots far to near (the nearest stays in `next`) and
// notes its hit leaf slots -- and a triangle phase -- each lane with noted
// leaves tests one of them. The lanes of a warp meet again before the
// triangle phase, so the warp runs it once per iteration for all of its
// lanes. A lane visits no node while it has untested leaves, so every node
// is entered with the t the reference-order loop would have after the
// previous node's leaves; only the order among one node's leaves (slot
// order here) differs, which can change the winner among triangles hit at
// exactly the same t.
//
// Rays the compact walk does not take -- a zero or non-finite component, an
// inverse direction beyond kQuantRange, an origin beyond kCompactRange, a
// node flagged out of range or a leaf of more than 32,767 primitives on the
// way or (GATES) a hit on a triangle
// flagged kTriEscape, see build_mbvh -- are appended to `deferred`
// and traced afterwards by k_trace_mbvh over the exact Mbvh.
// Nine resident blocks per SM (56 registers, 36 warps, no spills): eight are 5 %
// slower, ten (48 registers) spill and take 1.85 times as long.
//
// WSTATS: per-ray counts of this walk in a.walk_stats (traversal-tree node
// visits, triangle tests, 1 if the ray was handed to the exact walk).
template <int STACK, bool GATES, bool WSTATS>
__global__ void __launch_bounds__(kBlock, 9) k_trace_compact(TraceArgs a, unsigned int* work, uint32_t* deferred,
                                                           unsigned int* deferred_count) {
  RayState ray;
  float hu = 0.0f, hv = 0.0f;
  int32_t prim = -1;
  uint32_t w_visits = 0, w_tests = 0;
  int32_t stack[STACK];
  int sp = -1;
  int32_t next = -1;
  // the last visited node's hit leaf slots not yet tested, as bits of their
  // slots in lch / lct (first primitive slot, count)
  uint32_t pend = 0;
  int32_t lch[4] = {0, 0, 0, 0};
  uint32_t lct[2] = {0, 0};
  uint32_t r = 0;
  bool active = false;
  WarpPool pool;
  const uint32_t batch = a.ray_batch ? a.ray_batch : kPoolBatch;
  const uint32_t ray_count = (uint32_t)a.ray_count;
  auto write_stats = [&](uint32_t handed_on) {
    if (WSTATS) {
      a.walk_stats[3 * (size_t)r + 0] = w_visits;
      a.walk_stats[3 * (size_t)r + 1] = w_tests;
      a.walk_stats[3 * (size_t)r + 2] = handed_on;
    }
  };
  auto finish = [&]() {
    a.hits[r] = make_float4(ray.t, hu, hv, __int_as_float(prim));
    write_stats(0u);
    active = false;
  };
  auto defer = [&]() {
    deferred[atomicAdd(deferred_count, 1u)] = r;
    write_stats(1u);
    active = false;
  };
  auto start_ray = [&](uint32_t rr) {
    r = a.order ? __ldg(a.order + rr) : rr;
    ray = load_ray(a.rays, r, a.t_max);
    hu = hv = 0.0f;
    prim = -1;
    sp = -1;
    pend = 0;
    w_visits = w_tests = 0;
    if (!compact_root(a, r, next)) {
      finish();
      return;
    }
    if (!compact_ray(ray)) {
      defer();
      return;
    }
    active = true;
  };
  for (;;) {
    // refill once four lanes are idle: the ray set-up runs for the refilled
    // lanes only (and finds each ray's mesh in a forest). Two idle lanes: 64
    // meshes 7.67 instead of 7.33 ms, camera rays over 200k triangles +2 %,
    // incoherent rays +1 %; eight: incoherent +3 %.
    uint32_t amask = __ballot_sync(0xffffffffu, active);
    if (!pool.exhausted && __popc(amask) <= 28) {
      pool.refill<2>(active, batch, ray_count, work, start_ray);
      amask = __ballot_sync(0xffffffffu, active);
    }
    if (!amask) {
      if (pool.exhausted) break;
      continue;
    }
    if (!active) continue;
    // ---- node phase (no early exits: the lanes of amask meet below)
    if (pend == 0) {
      const int32_t current = next >= 0 ? next : stack[sp--];
      next = -1;
      if ((uint32_t)current >= a.q_count) {
        atomicOr(a.status, kStatusBadIndex);
        active = false;
      } else {
        const float* qn = reinterpret_cast<const float*>(a.qnodes + current);
        float h0[8], h1[8];
        ld8(qn, h0);
        ld8(qn + 8, h1);
        if (WSTATS) ++w_visits;
        const uint32_t flags = __float_as_uint(h0[3]) >> 24;
        if (flags & kQFlagOutOfRange) {
          defer();
        } else {
          float key[4];
          int32_t ich[4];
          bool large = false;
          if (!flags) slot_keys_q(h0, h1, ray, key, ich, pend, lch, lct);
          else slot_keys_exact(a.qexact + current, ray, key, ich, pend, lch, lct, large);
          // the nearest stays in `next`, the others are pushed far to near
          const float inf = __int_as_float(0x7f800000);
          const bool k1 = key[1] < inf, k2 = key[2] < inf, k3 = key[3] < inf;
          if (key[0] < inf) next = ich[0];
          sp += (k1 ? 1 : 0) + (k2 ? 1 : 0) + (k3 ? 1 : 0);
          if (sp >= STACK || large) {
            if (large) {
              defer();
            } else {
              atomicOr(a.status, kStatusStackOverflow);
              prim = -2;
              finish();
            }
          } else {
            if (k1) stack[sp] = ich[1];
            if (k2) stack[sp - 1] = ich[2];
            if (k3) stack[sp - 2] = ich[3];
          }
        }
      }
    }
    __syncwarp(amask);
    // ---- triangle phase
    if (active && pend) {
      const uint32_t i = __ffs(pend) - 1;
      pend &= pend - 1u;
      const int32_t lf = i == 0 ? lch[0] : (i == 1 ? lch[1] : (i == 2 ? lch[2] : lch[3]));
      const uint32_t cw = i < 2 ? lct[0] : lct[1];
      const int32_t count = (int32_t)((i & 1u) ? cw >> 16 : cw & 0xffffu);
      if (lf < 0 || (uint32_t)lf + (uint32_t)count > a.prim_count) {
        atomicOr(a.status, kStatusBadIndex);
        active = false;
      } else {
        for (int32_t j = 0; j < count; ++j) {
          const float4* tri = a.tris + kTriFloat4 * (size_t)(lf + j);
          if (WSTATS) ++w_tests;
          if (mt_test(tri, ray, hu, hv, prim) && GATES && (__float_as_uint(__ldg(&tri[1].w)) & kTriEscape)) {
            defer();  // an escaped triangle is hit: its hits are the exact walk's
            break;
          }
        }
      }
    }
    if (active && pend == 0 && next < 0 && sp < 0) finish();
  }
}

// One lane's slot of a compact node: the node's grid and the slot's near and
// far bounds as floats q * 2^-133 (see qbyte), picked by address.
struct LaneSlot {
  float4 head;
  uint32_t nx, fx, ny, fy, nz, fz;
  int32_t child, count;
  __device__ __forceinline__ void load(const DQNode* n, const RayState& ray, uint32_t l) {
    const uint8_t* node = reinterpret_cast<const uint8_t*>(n);
    const uint8_t* b = node + 16 + l;
    head = __ldg(reinterpret_cast<const float4*>(node));
    nx = __ldg(b + (ray.ix < 0.0f ? 4 : 0));
    fx = __ldg(b + (ray.ix < 0.0f ? 0 : 4));
    ny = __ldg(b + (ray.iy < 0.0f ? 12 : 8));
    fy = __ldg(b + (ray.iy < 0.0f ? 8 : 12));
    nz = __ldg(b + (ray.iz < 0.0f ? 20 : 16));
    fz = __ldg(b + (ray.iz < 0.0f ? 16 : 20));
    child = __ldg(reinterpret_cast<const int32_t*>(node + 40) + l);
    count = __ldg(reinterpret_cast<const int16_t*>(node + 56) + l);
  }
};

// k_trace_compact's walk, four lanes per ray, for few rays: every lane reads
// its own slot of a node and, where it is a leaf, tests it. The next node is
// popped and its slots are asked for before the leaves are tested.
template <bool GATES>
__global__ void __launch_bounds__(kBlock) k_trace_compact4(TraceArgs a, uint32_t warps, uint32_t* deferred,
                                                          unsigned int* deferred_count) {
  __shared__ int32_t s_stack[kBlock / 4][kStack];
  const FourLanes q;
  int32_t* stack = s_stack[threadIdx.x >> 2];
  const uint32_t warp = blockIdx.x * (kBlock / 32u) + (threadIdx.x >> 5);
  const float inf = __int_as_float(0x7f800000);
  RayState ray;
  float hu = 0.0f, hv = 0.0f;
  int32_t prim = -1, current = -1;  // the node whose slots are in `slot`
  int sp = -1;
  bool active = false;
  LaneSlot slot;
  // asks for the slots of `current`; false (the ray ends) when it is no node
  auto fetch = [&]() {
    if ((uint32_t)current >= a.q_count) {
      if (q.l == 0u) atomicOr(a.status, kStatusBadIndex);
      active = false;
    } else {
      slot.load(a.qnodes + current, ray, q.l);
    }
  };
  uint32_t r = 0;
  auto defer = [&]() {
    if (q.l == 0u) deferred[atomicAdd(deferred_count, 1u)] = r;
    active = false;
  };
  for (size_t i = warp < warps ? warp + (size_t)warps * (q.first >> 2) : a.ray_count;;) {
    if (!active && i < a.ray_count) {
      r = a.order ? __ldg(a.order + i) : (uint32_t)i;
      i += 8u * (size_t)warps;
      ray = load_ray(a.rays, r, a.t_max);
      hu = hv = 0.0f;
      prim = -1;
      sp = -1;
      active = compact_root(a, r, current);
      if (!active) {
        if (q.l == 0u) a.hits[r] = make_float4(ray.t, 0.0f, 0.0f, __int_as_float(-1));
      } else if (!compact_ray(ray)) {
        defer();
      } else {
        fetch();
      }
    }
    if (!__any_sync(0xffffffffu, active)) {
      if (!__any_sync(0xffffffffu, i < a.ray_count)) break;
      continue;
    }
    bool hit = false, inner = false, large = false;
    float key = inf;
    int32_t child = -1, count = -1;
    if (active) {
      const float4 head = slot.head;
      child = slot.child;
      count = slot.count;
      const uint32_t exps = __float_as_uint(head.w), flags = exps >> 24;
      float tn, tx, t;
      if (flags == 0u) {  // slot_keys_q
        const float sx = __uint_as_float(((exps & 0xffu) << 23) + kStepBias);
        const float sy = __uint_as_float(((exps >> 8 & 0xffu) << 23) + kStepBias);
        const float sz = __uint_as_float(((exps >> 16 & 0xffu) << 23) + kStepBias);
        const float ax = sx * ray.ix, bx = (head.x - ray.ox) * ray.ix * kKeyScale;
        const float ay = sy * ray.iy, by = (head.y - ray.oy) * ray.iy * kKeyScale;
        const float az = sz * ray.iz, bz = (head.z - ray.oz) * ray.iz * kKeyScale;
        tn = fmaxf(fmaf(__uint_as_float(slot.nx << 16), ax, bx),
                   fmaxf(fmaf(__uint_as_float(slot.ny << 16), ay, by), fmaf(__uint_as_float(slot.nz << 16), az, bz)));
        tx = fminf(fmaf(__uint_as_float(slot.fx << 16), ax, bx),
                   fminf(fmaf(__uint_as_float(slot.fy << 16), ay, by), fmaf(__uint_as_float(slot.fz << 16), az, bz)));
        t = ray.t * kKeyScale;
      } else {  // slot_keys_exact
        const float* n = reinterpret_cast<const float*>(a.qexact + current) + q.l;
        const float tx0 = (__ldg(n) - ray.ox) * ray.ix, tx1 = (__ldg(n + 4) - ray.ox) * ray.ix;
        const float ty0 = (__ldg(n + 8) - ray.oy) * ray.iy, ty1 = (__ldg(n + 12) - ray.oy) * ray.iy;
        const float tz0 = (__ldg(n + 16) - ray.oz) * ray.iz, tz1 = (__ldg(n + 20) - ray.oz) * ray.iz;
        child = __float_as_int(__ldg(n + 24));
        count = __float_as_int(__ldg(n + 28));
        large = count > 32767;
        tn = fmaxf(fminf(tx0, tx1), fmaxf(fminf(ty0, ty1), fminf(tz0, tz1)));
        tx = fminf(fmaxf(tx0, tx1), fminf(fmaxf(ty0, ty1), fmaxf(tz0, tz1)));
        t = ray.t;
      }
      hit = tx >= tn && tx >= 0.0f && tn < t && child >= 0;
      inner = hit && count < 0;
      if (inner) key = tn;
      large = large || (flags & kQFlagOutOfRange);
    }
    if (q.ballot(large)) {  // the exact walk's
      if (active) defer();
      hit = inner = false;
      key = inf;
    }
    // sort_slots over the four lanes
    int32_t near_child = child;
    auto exchange = [&](uint32_t with) {
      const float ok = q.from(key, with);
      const int32_t oc = q.from(near_child, with);
      if (q.l < with ? ok < key : (q.l > with && key < ok)) {
        key = ok;
        near_child = oc;
      }
    };
    exchange(q.l ^ 1u);
    exchange(q.l ^ 2u);
    exchange(q.l == 1u ? 2u : (q.l == 2u ? 1u : q.l));
    const int n = __popc(q.ballot(key < inf));
    const int32_t nearest = q.from(near_child, 0);
    bool done = false;
    int32_t next = -1;
    if (n > 0) {
      next = nearest;
      if (sp + n - 1 >= kStack) {
        if (q.l == 0u) atomicOr(a.status, kStatusStackOverflow);
        prim = -2;
        done = true;
      } else {
        if (q.l >= 1u && (int)q.l < n) stack[sp + n - (int)q.l] = near_child;
        sp += n - 1;
      }
    }
    __syncwarp();
    const bool leaf = hit && !inner && !done;
    if (active && !done) {
      current = next;
      if (next < 0 && sp >= 0) current = stack[sp--];
      if (current >= 0) fetch();
    }
    if (__any_sync(0xffffffffu, leaf)) {
      const float entry = ray.t;
      float u = hu, v = hv, escaped = inf;
      int32_t p = prim;
      bool bad = false;
      if (leaf) {
        bad = (uint32_t)child + (uint32_t)count > a.prim_count;
        if (bad) atomicOr(a.status, kStatusBadIndex);
        for (int32_t j = 0; !bad && j < count; ++j) {
          const float4* tri = a.tris + kTriFloat4 * (size_t)(child + j);
          if (mt_test(tri, ray, u, v, p) && GATES && (__float_as_uint(__ldg(&tri[1].w)) & kTriEscape)) escaped = ray.t;
        }
      }
      float best, before;
      const int w = first_nearest<false>(q, ray.t, entry, best, before);
      const uint32_t src = w < 0 ? q.l : (uint32_t)w;
      const float wt = q.from(ray.t, src), wu = q.from(u, src), wv = q.from(v, src);
      const int32_t wp = q.from(p, src);
      ray.t = entry;
      if (w >= 0) {
        ray.t = wt;
        hu = wu;
        hv = wv;
        prim = wp;
      }
      const uint32_t bads = q.ballot(bad);
      const uint32_t escapes = q.ballot(GATES && escaped < before);
      if (active && bads) active = false;
      else if (active && escapes) defer();  // an escaped triangle is hit: its hits are the exact walk's
    }
    if (active && (done || current < 0)) {
      if (q.l == 0u) a.hits[r] = make_float4(ray.t, hu, hv, __int_as_float(prim));
      active = false;
    }
  }
}

// Aabb::intersect (src/aabb.rs:145-181): far t or miss; t_min fixed at 1e-4.
__device__ __forceinline__ bool slab_far(const DAabb& b, const RayState& r, float& out) {
  float ray_min = ((r.sx ? b.max[0] : b.min[0]) - r.ox) * r.ix;
  float ray_max = ((r.sx ? b.min[0] : b.max[0]) - r.ox) * r.ix;
  const float y_min = ((r.sy ? b.max[1] : b.min[1]) - r.oy) * r.iy;
  const float y_max = ((r.sy ? b.min[1] : b.max[1]) - r.oy) * r.iy;
  if ((ray_min > y_max) || (y_min > ray_max)) return false;
  if (y_min > ray_min) ray_min = y_min;
  if (y_max < ray_max) ray_max = y_max;
  const float z_min = ((r.sz ? b.max[2] : b.min[2]) - r.oz) * r.iz;
  const float z_max = ((r.sz ? b.min[2] : b.max[2]) - r.oz) * r.iz;
  if ((ray_min > z_max) || (z_min > ray_max)) return false;
  if (z_max < ray_max) ray_max = z_max;
  if (ray_max > 1e-4f) {
    out = ray_max;
    return true;
  }
  return false;
}

// BvhIndexIterator::next (src/iter_indices.rs:66-107) for one ray: a step
// is one pop; a leaf's primitives are tested, an interior node's two
// children are tested with the far-t slab test (which never culls by t) and
// pushed in sort_nodes order. Stack entries hold the node's (left_first,
// count), read when its parent loaded both children (two 256-bit loads of
// the adjacent pair), so a pop needs no node load.
template <bool ANY_HIT, bool STATS>
__device__ __forceinline__ void trace_one_bvh(const TraceArgs& a, size_t r) {
  RayState ray = load_ray(a.rays, r, a.t_max);
  float hu = 0.0f, hv = 0.0f;
  int32_t prim = -1;
  uint32_t visits = 0, tests = 0, max_depth = 0;
  const bool nan = (ray.ox != ray.ox) || (ray.oy != ray.oy) || (ray.oz != ray.oz) || (ray.dx != ray.dx) ||
                   (ray.dy != ray.dy) || (ray.dz != ray.dz);
  int2 stack[kStack];
  int sp = -1;
  if (a.node_count > 0 && !nan) {
    const DAabb root = load_aabb(a.nodes);
    stack[0] = make_int2(root.left_first, root.count);
    sp = 0;
  }
  while (sp >= 0) {
    const int2 e = stack[sp--];
    const int32_t lf = e.x, count = e.y;
    if (count > -1) {
      if (lf < 0 || (uint32_t)lf + (uint32_t)count > a.prim_count) {
        atomicOr(a.status, kStatusBadIndex);
        break;
      }
      bool stop = false;
      for (int32_t j = 0; j < count; ++j) {
        if (STATS) ++tests;
        if (mt_test(a.tris + kTriFloat4 * (size_t)(lf + j), ray, hu, hv, prim) && ANY_HIT) {
          stop = true;
          break;
        }
      }
      if (stop) break;
    } else if (lf > -1) {
      if (STATS) ++visits;
      if ((uint32_t)lf + 1u >= a.node_count) {
        atomicOr(a.status, kStatusBadIndex);
        break;
      }
      float l8[8], r8[8];
      ld8(reinterpret_cast<const float*>(a.nodes + lf), l8);
      ld8(reinterpret_cast<const float*>(a.nodes + lf + 1), r8);
      DAabb lb, rb;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lb.min[k] = l8[k];
        lb.max[k] = l8[4 + k];
        rb.min[k] = r8[k];
        rb.max[k] = r8[4 + k];
      }
      const int2 le = make_int2(__float_as_int(l8[7]), __float_as_int(l8[3]));
      const int2 re = make_int2(__float_as_int(r8[7]), __float_as_int(r8[3]));
      float lt = 0.0f, rt = 0.0f;
      const bool lh = slab_far(lb, ray, lt);
      const bool rh = slab_far(rb, ray, rt);
      if (sp + 2 >= kStack) {
        atomicOr(a.status, kStatusStackOverflow);
        prim = -2;
        break;
      }
      if (lh && rh) {
        if (lt < rt) { stack[++sp] = le; stack[++sp] = re; }
        else { stack[++sp] = re; stack[++sp] = le; }
      } else if (lh) {
        stack[++sp] = le;
      } else if (rh) {
        stack[++sp] = re;
      }
      if (STATS && (uint32_t)(sp + 1) > max_depth) max_depth = (uint32_t)(sp + 1);
    }
  }
  a.hits[r] = make_float4(ray.t, hu, hv, __int_as_float(prim));
  if (STATS) {
    a.stats[3 * (size_t)r + 0] = visits;
    a.stats[3 * (size_t)r + 1] = tests;
    a.stats[3 * (size_t)r + 2] = max_depth;
  }
}

// Warps take 32 consecutive rays at a time (adjacent camera rays walk the
// same nodes in step).
template <bool ANY_HIT, bool STATS>
__global__ void __launch_bounds__(kBlock) k_trace_bvh(TraceArgs a, unsigned int* work) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned int base = 0;
    if (lane == 0) base = atomicAdd(work, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if ((size_t)base >= a.ray_count) break;
    const size_t r = (size_t)base + lane;
    if (r < a.ray_count) trace_one_bvh<ANY_HIT, STATS>(a, r);
  }
}

// ------------------------------------------------------------------ candidate lists
// The primitives the reference's index iterators yield for a ray when the
// caller's callback leaves t unchanged: MbvhIndexIterator
// (src/iter_indices.rs:212-313) or BvhIndexIterator (:18-107) over the exact
// nodes, in yield order. This is the device form of intersect /
// intersect_mbvh with a user callback (rtbvh_ffi/src/lib.rs:551-581,
// 700-731) for primitives whose test the library does not know: the caller
// tests the listed primitives in its own kernel. One ray per thread.
template <bool MBVH>
__global__ void __launch_bounds__(kBlock) k_candidates(CandArgs a) {
  const size_t stride = (size_t)gridDim.x * kBlock;
  for (size_t r = (size_t)blockIdx.x * kBlock + threadIdx.x; r < a.ray_count; r += stride) {
    const RayState ray = load_ray(a.rays, r, a.t_max);
    uint32_t n = 0;
    bool bad = false;
    auto yield_range = [&](int32_t lf, int32_t count) {
      if (lf < 0 || (uint32_t)lf + (uint32_t)count > a.prim_count) {
        atomicOr(a.status, kStatusBadIndex);
        bad = true;
        return;
      }
      for (int32_t j = 0; j < count; ++j) {
        if (a.out && n < a.max_per_ray) a.out[r * a.max_per_ray + n] = __ldg(a.indices + lf + j);
        ++n;
      }
    };
    int32_t stack[kStack];
    int sp = -1;
    if (MBVH) {
      if (a.node_count > 0) {
        const bool fast = finite_ray(ray);
        int32_t current = 0;
        for (;;) {
          uint32_t mask, ids;
          int4 children, counts;
          if (fast) quad_intersect<true>(a.mnodes + current, ray, mask, ids, children, counts);
          else quad_intersect<false>(a.mnodes + current, ray, mask, ids, children, counts);
          for (int i = 0; i < 4 && !bad; ++i) {
            const uint32_t id = (ids >> (2 * (3 - i))) & 3u;
            if (!((mask >> id) & 1u)) continue;
            const int32_t count = sel4(counts, id), lf = sel4(children, id);
            if (count > -1) {
              yield_range(lf, count);
            } else if (lf > -1) {
              if (sp + 1 >= kStack) {
                atomicOr(a.status, kStatusStackOverflow);
                bad = true;
                break;
              }
              stack[++sp] = lf;
            }
          }
          if (bad || sp < 0) break;
          current = stack[sp--];
          if ((uint32_t)current >= a.node_count) {
            atomicOr(a.status, kStatusBadIndex);
            bad = true;
            break;
          }
        }
      }
    } else {
      const bool nan = (ray.ox != ray.ox) || (ray.oy != ray.oy) || (ray.oz != ray.oz) || (ray.dx != ray.dx) ||
                       (ray.dy != ray.dy) || (ray.dz != ray.dz);
      sp = (a.node_count == 0 || nan) ? -1 : 0;
      stack[0] = 0;
      while (sp >= 0 && !bad) {
        const int32_t ni = stack[sp--];
        if ((uint32_t)ni >= a.node_count) {
          atomicOr(a.status, kStatusBadIndex);
          bad = true;
          break;
        }
        const DAabb node = load_aabb(a.nodes + ni);
        if (node.count > -1) {
          yield_range(node.left_first, node.count);
        } else if (node.left_first > -1) {
          const int32_t lf = node.left_first;
          if ((uint32_t)lf + 1u >= a.node_count) {
            atomicOr(a.status, kStatusBadIndex);
            bad = true;
            break;
          }
          float lt = 0.0f, rt = 0.0f;
          const bool lh = slab_far(load_aabb(a.nodes + lf), ray, lt);
          const bool rh = slab_far(load_aabb(a.nodes + lf + 1), ray, rt);
          if (sp + 2 >= kStack) {
            atomicOr(a.status, kStatusStackOverflow);
            bad = true;
            break;
          }
          if (lh && rh) {
            if (lt < rt) { stack[++sp] = lf; stack[++sp] = lf + 1; }
            else { stack[++sp] = lf + 1; stack[++sp] = lf; }
          } else if (lh) {
            stack[++sp] = lf;
          } else if (rh) {
            stack[++sp] = lf + 1;
          }
        }
      }
    }
    a.counts[r] = bad ? 0xffffffffu : n;
  }
}

// ------------------------------------------------------------------ ray order
// Incoherent rays are traced in an order that groups rays with nearby
// origins and similar directions, so that the lanes of a warp walk similar
// nodes (fewer distinct cache lines per warp load, more L1 hits). Each ray's
// traversal is unchanged; only the assignment of rays to lanes differs, and
// hits are written to the ray's own slot.

__global__ void __launch_bounds__(256) k_ray_origin_bounds(const float* __restrict__ rays, size_t n,
                                                           uint32_t* __restrict__ acc) {
  float mn[3] = {3.4e38f, 3.4e38f, 3.4e38f}, mx[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float2* p = reinterpret_cast<const float2*>(rays + 6 * i);
    const float2 a = __ldg(p), b = __ldg(p + 1);
    const float o[3] = {a.x, a.y, b.x};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (isfinite(o[k])) {
        mn[k] = fminf(mn[k], o[k]);
        mx[k] = fmaxf(mx[k], o[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], off));
      mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], off));
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      atomicMin(acc + k, float_to_ordered(mn[k]));
      atomicMax(acc + 3 + k, float_to_ordered(mx[k]));
    }
  }
}

__device__ __forceinline__ uint32_t spread3_bits(uint32_t v) {
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}
__device__ __forceinline__ uint32_t spread2_bits(uint32_t v) {
  v = (v | (v << 8)) & 0x00FF00FFu;
  v = (v | (v << 4)) & 0x0F0F0F0Fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}
__device__ __forceinline__ uint32_t quant6(float x) {  // x in [0, 1]
  float q = x * 64.0f;
  return q >= 63.0f ? 63u : (q > 0.0f ? (uint32_t)q : 0u);
}

// key = Morton(origin cell, 6 bits per axis) << 12 | Morton(octahedral
// direction, 6 bits per coordinate)
__global__ void __launch_bounds__(256) k_ray_keys(const float* __restrict__ rays, size_t n,
                                                  const uint32_t* __restrict__ acc, uint32_t* __restrict__ keys,
                                                  uint32_t* __restrict__ vals) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float lo[3], inv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = ordered_to_float(__ldg(acc + k));
    const float ext = ordered_to_float(__ldg(acc + 3 + k)) - lo[k];
    inv[k] = ext > 0.0f ? 1.0f / ext : 0.0f;
  }
  const float2* p = reinterpret_cast<const float2*>(rays + 6 * i);
  const float2 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
  const float o[3] = {a.x, a.y, b.x};
  const float d[3] = {b.y, c.x, c.y};
  uint32_t oc[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) oc[k] = quant6((o[k] - lo[k]) * inv[k]);
  const float l1 = fabsf(d[0]) + fabsf(d[1]) + fabsf(d[2]);
  float u = 0.0f, v = 0.0f;
  if (l1 > 0.0f && isfinite(l1)) {
    u = d[0] / l1;
    v = d[1] / l1;
    if (d[2] < 0.0f) {
      const float uu = (1.0f - fabsf(v)) * (u >= 0.0f ? 1.0f : -1.0f);
      const float vv = (1.0f - fabsf(u)) * (v >= 0.0f ? 1.0f : -1.0f);
      u = uu;
      v = vv;
    }
  }
  const uint32_t du = quant6(u * 0.5f + 0.5f), dv = quant6(v * 0.5f + 0.5f);
  const uint32_t ko = spread3_bits(oc[0]) | (spread3_bits(oc[1]) << 1) | (spread3_bits(oc[2]) << 2);
  keys[i] = (ko << 12) | spread2_bits(du) | (spread2_bits(dv) << 1);
  vals[i] = (uint32_t)i;
}

// Persistent grid: resident blocks per SM (occupancy, capped by
// blocks_per_sm) on every SM, no more blocks than the rays need.
template <class K>
unsigned persistent_grid(K kern, const TraceArgs& a, size_t rays_per_block = kBlock) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, 0);
  if (per_sm < 1) per_sm = 1;
  if (a.blocks_per_sm > 0 && (int)a.blocks_per_sm < per_sm) per_sm = (int)a.blocks_per_sm;
  size_t grid = (size_t)sm_count() * per_sm;
  const size_t need = (a.ray_count + rays_per_block - 1) / rays_per_block;
  if (grid > need) grid = need;
  return (unsigned)grid;
}

template <bool MBVH, bool ANY_HIT, bool STATS>
cudaError_t launch3(const TraceArgs& a, cudaStream_t s, unsigned int* work) {
  auto kern = MBVH ? k_trace_mbvh<ANY_HIT, STATS> : k_trace_bvh<ANY_HIT, STATS>;
  kern<<<persistent_grid(kern, a), kBlock, 0, s>>>(a, work);
  return cudaGetLastError();
}

// Closest hit through the compact traversal tree, then the rays it deferred
// over the exact Mbvh. counters: [0] compact ray counter, [1] deferred rays,
// [2] exact ray counter (zeroed).
template <bool WSTATS>
auto compact_kernel(const TraceArgs& a) {
  return a.q_gates ? (a.stack_limit == 32   ? k_trace_compact<32, true, WSTATS>
                      : a.stack_limit == 48 ? k_trace_compact<48, true, WSTATS>
                                            : k_trace_compact<64, true, WSTATS>)
                   : (a.stack_limit == 32   ? k_trace_compact<32, false, WSTATS>
                      : a.stack_limit == 48 ? k_trace_compact<48, false, WSTATS>
                                            : k_trace_compact<64, false, WSTATS>);
}

// Launches of few rays with no launch shape asked for: four lanes per ray.
bool few_rays(const TraceArgs& a) {
  return a.ray_count <= (a.any_hit ? kFewAny : kFewClosest) && a.ray_batch == 0 && a.blocks_per_sm == 0 &&
         (a.stack_limit == 0 || a.stack_limit == (uint32_t)kStack);
}

template <bool ANY_HIT, int CULL>
cudaError_t launch_few(const TraceArgs& a, cudaStream_t s) {
  const uint32_t warps = few_warps((uint32_t)a.ray_count, (uint32_t)sm_count());
  k_trace_mbvh4<ANY_HIT, CULL><<<(warps + 3u) / 4u, kBlock, 0, s>>>(a, warps);
  return cudaGetLastError();
}

cudaError_t launch_compact(const TraceArgs& a, cudaStream_t s, unsigned int* counters, uint32_t* deferred) {
  if (few_rays(a) && !a.walk_stats) {
    const uint32_t warps = few_warps((uint32_t)a.ray_count, (uint32_t)sm_count());
    auto kern = a.q_gates ? k_trace_compact4<true> : k_trace_compact4<false>;
    kern<<<(warps + 3u) / 4u, kBlock, 0, s>>>(a, warps, deferred, counters + 1);
  } else {
    auto kern = a.walk_stats ? compact_kernel<true>(a) : compact_kernel<false>(a);
    kern<<<persistent_grid(kern, a), kBlock, 0, s>>>(a, counters, deferred, counters + 1);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  TraceArgs b = a;
  b.order = deferred;
  b.ray_count_dev = counters + 1;
  // at most 32 rays per refill (the kernel takes fewer when few rays were
  // deferred)
  b.ray_batch = 32;
  b.sms = (uint32_t)sm_count();
  auto rest = b.tboxes ? k_trace_mbvh<false, false, kCullSubtree, true> : k_trace_mbvh<false, false, kCullNone, true>;
  rest<<<persistent_grid(rest, b, kBlock / 4), kBlock, 0, s>>>(b, counters + 2);
  return cudaGetLastError();
}

template <bool MBVH>
cudaError_t launch_any(const TraceArgs& a0, cudaStream_t s) {
  if (a0.ray_count == 0) return cudaSuccess;
  // ray indices and the work counter are 32-bit; after the last batch every
  // warp adds one more ray_batch (<= 4096) to the counter, which must not wrap
  if (a0.ray_count > 0xffffffffull - (1ull << 25) || a0.ray_batch > 4096u) return cudaErrorInvalidValue;
  if (a0.stack_limit != 0 && a0.stack_limit != 32 && a0.stack_limit != 48 && a0.stack_limit != 64)
    return cudaErrorInvalidValue;
  TraceArgs a = a0;
  // any hit: most walks end after a few nodes, so refills are frequent and
  // larger pools cost fewer counter atomics (128: 34.0 against 28.7 Grays/s
  // with 32 on the 1M incoherent scene's occlusion rays), but not so large
  // that a launch has fewer pools than warps (131,072 shadow rays over 300k
  // clustered triangles: 301 us with pools of 32, 500 with 128)
  const bool few = few_rays(a);
  if (a.any_hit && a.ray_batch == 0) {
    const size_t even = a.ray_count / ((size_t)sm_count() * 32u);  // rays per resident warp
    a.ray_batch = even < 32u ? 32u : (even < 128u ? (uint32_t)even : 128u);
  }
  Scratch<unsigned int> work;
  Scratch<uint32_t> keys, order, acc, deferred;
  Scratch<char> sort_temp;
  cudaError_t e;
  if ((e = work.alloc(4, s)) || (e = cudaMemsetAsync(work.ptr, 0, 4 * sizeof(unsigned int), s))) return e;
  if (MBVH && a.order == nullptr && a.reorder && a.ray_count < (1u << 30)) {
    const size_t n = a.ray_count;
    const size_t tb = radix_sort_temp_bytes(n);
    if ((e = keys.alloc(n, s)) || (e = order.alloc(n, s)) || (e = acc.alloc(8, s)) || (e = sort_temp.alloc(tb, s)))
      return e;
    const uint32_t init[8] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u, 0u, 0u};
    if ((e = cudaMemcpyAsync(acc.ptr, init, sizeof(init), cudaMemcpyHostToDevice, s))) return e;
    unsigned blocks = (unsigned)((n + 255) / 256);
    const unsigned cap = (unsigned)sm_count() * 8u;
    k_ray_origin_bounds<<<blocks < cap ? blocks : cap, 256, 0, s>>>(a.rays, n, acc.ptr);
    k_ray_keys<<<blocks, 256, 0, s>>>(a.rays, n, acc.ptr, keys.ptr, order.ptr);
    if ((e = radix_sort_pairs(keys.ptr, order.ptr, n, 30, sort_temp.ptr, tb, a.status, s))) return e;
    a.order = order.ptr;
  }
  const bool st = a.stats != nullptr;
  if (a.any_hit && MBVH && !st) {
    const bool behind = a.root_covers && a.edges && a.quads_cover;
    const bool subtree = a.root_covers && a.edges && !behind && a.tboxes;
    if (few) {
      e = behind ? launch_few<true, kCullBehind>(a, s)
                 : (subtree ? launch_few<true, kCullSubtree>(a, s) : launch_few<true, kCullNone>(a, s));
    } else {
      auto kern = behind ? k_trace_mbvh<true, false, kCullBehind>
                         : (subtree ? k_trace_mbvh<true, false, kCullSubtree> : k_trace_mbvh<true, false>);
      kern<<<persistent_grid(kern, a), kBlock, 0, s>>>(a, work.ptr);
      e = cudaGetLastError();
    }
  } else if (a.any_hit) e = st ? launch3<MBVH, true, true>(a, s, work.ptr) : launch3<MBVH, true, false>(a, s, work.ptr);
  else if (st) e = launch3<MBVH, false, true>(a, s, work.ptr);
  else if (MBVH && a.qnodes && a.q_count > 0) {
    if ((e = deferred.alloc(a.ray_count, s))) return e;
    e = launch_compact(a, s, work.ptr, deferred.ptr);
  } else if (MBVH && few) e = launch_few<false, kCullNone>(a, s);
  else e = launch3<MBVH, false, false>(a, s, work.ptr);
  return e;
}

}  // namespace

cudaError_t launch_trace_mbvh(const TraceArgs& a, cudaStream_t s) { return launch_any<true>(a, s); }
cudaError_t launch_trace_bvh(const TraceArgs& a, cudaStream_t s) { return launch_any<false>(a, s); }

cudaError_t launch_candidates(const CandArgs& a, bool mbvh, cudaStream_t s) {
  if (a.ray_count == 0) return cudaSuccess;
  auto kern = mbvh ? k_candidates<true> : k_candidates<false>;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, 0);
  if (per_sm < 1) per_sm = 1;
  size_t grid = (size_t)sm_count() * per_sm;
  const size_t need = (a.ray_count + kBlock - 1) / kBlock;
  if (grid > need) grid = need;
  kern<<<(unsigned)grid, kBlock, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace rtbvh
