// trace.cuh -- octree closest-hit / any-hit traversal and the primitive
// tests, as device functions shared by the ray-batch kernels (trace.cu) and
// the path tracer (wavefront.cu).
//
// Exactness.  Hit ids must equal the reference's bit for bit, so every
// float operation on this path is an explicit round-to-nearest intrinsic
// (__fadd_rn, __fmul_rn, ...): nothing can be contracted into an FMA whatever
// the compile flags, and each expression rounds as the reference's
// TVec/TPos code does when evaluated left to right in IEEE single precision.
//
// Traversal order.  The reference recurses (space/octree.cc:175-300): at a
// node it first tests the node's own surface list, then visits the children
// in the order i = 0,1,2,4,3,5,6,7 (bits swapped so the number of "far" bits
// never decreases) xor the ray's origin octant, each behind a per-axis gate,
// and each child call begins with a slab cull.  Here the recursion becomes an
// explicit stack: of the children that pass gate and cull *now* (at most 4 --
// a segment meets at most 4 octants) the first is entered directly and the
// others wait in one record; a closest-hit query's next entry is then culled
// again with the ray's *current* extent.  Because the ray only ever shrinks,
// the first test admits a superset, and the second decides as the recursion
// does at that point: with finite bounds whatever the gate closes the cull
// closes too, so the gate itself is evaluated again only where calls are
// counted or bounds may be NaN.  (An any-hit query's extent never changes: its
// entries are not tested again.)  Entries are taken in the recursion's order,
// so the set and order of surface tests -- and the surviving hit -- are the
// reference's.  The reference's negative-result
// cache (space/isec-cache.h) only skips re-testing a surface that already
// missed; a miss stays a miss for a ray that only shrinks, so omitting it
// changes work, not results.

#ifndef SNOG_TRACE_CUH
#define SNOG_TRACE_CUH

#include "snog_common.h"

namespace snog {

// -- exact float3 arithmetic ------------------------------------------------
__device__ __forceinline__ float3 xadd(float3 a, float3 b) {
  return f3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z));
}
__device__ __forceinline__ float3 xsub(float3 a, float3 b) {
  return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 xmul(float3 a, float s) {
  return f3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s));
}
__device__ __forceinline__ float xdot(float3 a, float3 b) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 xcross(float3 a, float3 b) {
  return f3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)),
            __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
            __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float xlen_sq(float3 a) { return xdot(a, a); }

constexpr float kEps = 1e-15f;   // geometry/coords.h:48

// tripar_intersects (geometry/tripar-isec.h:56-118) plus the t < t1 bound of
// the ray form (tripar-isec.h:158-170).
__device__ __forceinline__ bool tripar_hit(float3 corner, float3 e1, float3 e2, bool parallelogram,
                                           float3 o, float3 d, float t0, float t1, float &t,
                                           float &u, float &v) {
  float3 pvec = xcross(d, e2);
  float det = xdot(e1, pvec);
  if (det > -kEps && det < kEps) return false;
  float inv_det = __frcp_rn(det);   // = 1.0f / det, correctly rounded
  float3 tvec = xsub(o, corner);
  u = __fmul_rn(xdot(tvec, pvec), inv_det);
  if (u < 0.f || u > 1.f) return false;
  float3 qvec = xcross(tvec, e1);
  v = __fmul_rn(xdot(d, qvec), inv_det);
  if (parallelogram) {
    if (v < 0.f || v > 1.f) return false;
  } else {
    if (v < 0.f || __fadd_rn(u, v) > 1.f) return false;
  }
  t = __fmul_rn(xdot(e2, qvec), inv_det);
  return t > t0 && t < t1;
}

// tripar_hit evaluated to the end without early exits: the same
// operations and the same result, but a warp whose lanes would leave at
// different tests does not diverge.  What list rounds use (against early exits:
// the intersection batch +2.4 %; shadow rays of the terrain frame 51.2 -> 50.6
// ms, of a Cornell render 0.653 -> 0.623).
__device__ __forceinline__ bool tripar_hit_flat(float3 corner, float3 e1, float3 e2, bool parallelogram,
                                                float3 o, float3 d, float t0, float t1, float &t) {
  const float3 pvec = xcross(d, e2);
  const float det = xdot(e1, pvec);
  bool ok = !(det > -kEps && det < kEps);
  const float inv_det = __frcp_rn(det);
  const float3 tvec = xsub(o, corner);
  const float u = __fmul_rn(xdot(tvec, pvec), inv_det);
  ok = ok && !(u < 0.f || u > 1.f);
  const float3 qvec = xcross(tvec, e1);
  const float v = __fmul_rn(xdot(d, qvec), inv_det);
  ok = ok && !(v < 0.f || (parallelogram ? v > 1.f : __fadd_rn(u, v) > 1.f));
  t = __fmul_rn(xdot(e2, qvec), inv_det);
  return ok && t > t0 && t < t1;
}

// sphere_intersects + quadratic_roots (geometry/sphere-isec.h:35-94,
// geometry/quadratic-roots.h:28-66): the first root above t0, then < t1.
__device__ __forceinline__ bool sphere_hit(float3 center, float radius, float3 o, float3 d,
                                           float t0, float t1, float &t) {
  float3 oo = xsub(o, center);
  float a = xlen_sq(d);
  float b = __fmul_rn(2.0f, xdot(d, oo));
  float c = __fsub_rn(xlen_sq(oo), __fmul_rn(radius, radius));
  float r0, r1;
  int n;
  if (a == 0.f) {
    if (b == 0.f) return false;
    r0 = __fdiv_rn(-c, b);
    r1 = r0;
    n = 1;
  } else {
    float disc = __fsub_rn(__fmul_rn(b, b), __fmul_rn(__fmul_rn(4.0f, a), c));
    if (disc < 0.f) return false;
    float sq = __fsqrt_rn(disc);
    float q = __fdiv_rn(-__fadd_rn(b, (b < 0.f ? -sq : sq)), 2.0f);
    r0 = __fdiv_rn(q, a);
    if (q == 0.f) {
      r1 = r0;
      n = 1;
    } else {
      r1 = __fdiv_rn(c, q);
      n = 2;
      if (r0 > r1) {
        float tmp = r0;
        r0 = r1;
        r1 = tmp;
      }
    }
  }
  if (r0 > t0) {
    t = r0;
    return t < t1;
  }
  if (n == 2 && r1 > t0) {
    t = r1;
    return t < t1;
  }
  return false;
}

struct TraceCounters {
  uint32_t nodes;     // node calls (space_node_intersect_calls)
  uint32_t tests;     // surface tests (surface_intersects_tests, no neg. cache)
  uint32_t overflow;  // traversal stack was too small (result invalid)
};

// Child slot IDX of a node whose 8 child ids are in K0, K1, by selects (no
// dynamically indexed local array).
__device__ __forceinline__ uint32_t pick_child(uint4 k0, uint4 k1, uint32_t idx) {
  uint4 k = (idx & 4u) ? k1 : k0;
  uint32_t a = (idx & 1u) ? k.y : k.x;
  uint32_t b = (idx & 1u) ? k.w : k.z;
  return (idx & 2u) ? b : a;
}

// A primitive's 48-byte record (snog_common.h).
struct PrimRec {
  float4 a, b, c;
};

__device__ __forceinline__ PrimRec load_prim(const DevScene &s, uint32_t id) {
  const float4 *p = s.prims + 3 * size_t(id);
  return PrimRec{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
}

// Test a loaded primitive against the ray; closest queries shrink t1 on a
// hit (the surface's intersect / intersects methods, surface/mesh.cc:730-760,
// surface/sphere.cc:110-125, surface/tripar.cc:93-115).
__device__ __forceinline__ bool test_prim(const PrimRec &r, float3 o, float3 d, float t0, float &t1) {
  const float kind = r.a.w;
  float t;
  const bool hit = kind == float(PRIM_SPHERE)
                       ? sphere_hit(xyz(r.a), r.b.x, o, d, t0, t1, t)
                       : tripar_hit_flat(xyz(r.a), xyz(r.b), xyz(r.c), kind == float(PRIM_PARALLELOGRAM), o, d, t0,
                                         t1, t);
  if (hit) t1 = t;
  return hit;
}

// The pending children of one visited node, as one stack record: the
// node's lower bounds and half extents along the ray (a child's bounds are lo
// or mid = lo + half, and its lower bound + half, per axis), its first child's
// index, its child mask and the children not yet entered (by octant bits).
// One record per visited node with two or more qualifying children,
// instead of one entry per waiting child: a visit pushes at most once, and
// the stack holds at most one record per tree level.
struct StackRec {
  float4 a;   // lo.xyz, first child index
  float4 b;   // half.xyz, child mask | children still to enter << 8
};

// Threads per block of every trace kernel.
constexpr int kTraceBlock = 128;
// Blocks per SM the trace kernels are compiled for (register cap 64).
#ifndef SNOG_TRACE_MINBLOCKS
#define SNOG_TRACE_MINBLOCKS 8
#endif

// The newest kRing records of each thread's stack live in shared memory, as
// a ring; older ones spill to the thread's local-memory array.  Lanes of a
// warp sit at different stack depths, so a local-memory stack is read and
// written uncoalesced; the ring keeps the pushes and pops of a walk on chip
// (kRing * 32 bytes per thread, 16 KB per 128-thread block at kRing = 4).
#ifndef SNOG_RING
#define SNOG_RING 4
#endif
constexpr uint32_t kRing = SNOG_RING;

// This thread's first ring slot.  Part k (0, 1) of record position e of
// thread t is float4 (2 * e + k) * kTraceBlock + t: a warp touching one part
// of one position reads 512 contiguous bytes.
__device__ __forceinline__ float4 *ring_slots() {
  __shared__ float4 ring[2 * kRing * kTraceBlock];
  return ring + threadIdx.x;
}

// Each thread's current ray in shared memory, for the lanes that test its
// list entries (a list round would otherwise move 14 values by shuffles):
// uint4 k * kTraceBlock + threadIdx.x holds, for k = 0, 1, 2, (origin, t0),
// (direction, t1) and the scene's list-record pointer in x, y; z, w of the
// third belong to the list round: what the units of the warp's k-th owner need.
__device__ __forceinline__ uint4 *ray_slots() {
  __shared__ uint4 rays[3 * kTraceBlock];
  return rays;
}

constexpr uint32_t kSlowSlab = 8u;   // in Traversal::octant: slab bounds may be NaN
constexpr uint32_t kAnyHit = 16u;    // in Traversal::octant: an any-hit query
constexpr uint32_t kGateFlag = 32u;  // in Traversal::octant: the entry carries a parent gate,
constexpr uint32_t kGateShift = 6u;  //   whose octant bits start here
enum { kClosestOnly = 0, kAnyOnly = 1, kMixed = 2 };   // queries a trace kernel runs

__device__ __forceinline__ bool slab_open(float t0, float t1, float3 lo, float3 hi) {
  float min_t = fmax_ref(t0, fmax_ref(lo.x, fmax_ref(lo.y, lo.z)));
  float max_t = fmin_ref(t1, fmin_ref(hi.x, fmin_ref(hi.y, hi.z)));
  return !(min_t >= max_t);
}

// slab_open for bounds known to be NaN-free (finite slab, t0 and t1 not
// NaN): maxima and minima are then exact and associative, so fmaxf / fminf
// in any grouping decide the same as the reference's ordered ternaries.
__device__ __forceinline__ bool slab_open_finite(float t0, float t1, float3 lo, float3 hi) {
  return fmaxf(fmaxf(t0, lo.x), fmaxf(lo.y, lo.z)) < fminf(fminf(t1, hi.x), fminf(hi.y, hi.z));
}

// The parent's gate for a child with octant bits CB (parametric order), at
// the current extent: a "far" half needs t1 beyond the midpoint, a "near"
// half needs t0 before it (space/octree.cc:268-272).  For the far half the
// midpoint is the child's lower bound, for the near half its upper bound --
// the very same rounded sums the reference compares against.
__device__ __forceinline__ bool gate_open(uint32_t cb, float t0, float t1, float3 lo, float3 hi) {
  bool gx = (cb & 4) ? (t1 > lo.x) : (t0 < hi.x);
  bool gy = (cb & 2) ? (t1 > lo.y) : (t0 < hi.y);
  bool gz = (cb & 1) ? (t1 > lo.z) : (t0 < hi.z);
  return gx && gy && gz;
}

// The child of the waiting set VM (bit cb = the child with octant bits cb,
// x = 4, y = 2, z = 1, a set bit meaning the half the ray enters later) that
// the reference visits first: its order is 0,1,2,4,3,5,6,7, so 4 goes before 3.
__device__ __forceinline__ uint32_t first_child(uint32_t vm) {
  return (vm & 0x1fu) == 0x18u ? 4u : uint32_t(__ffs(vm)) - 1u;
}

// A resumable octree walk for one ray.  init() sets up the root's slab
// bounds (space/octree.cc:119-135); node_step() processes the current octree
// entry as one call of the reference's recursive function does: parent gate,
// slab cull, then the node's surface list (left pending in [lp, lend) for
// list_round) and the children, the first of which -- or else the next child
// waiting on the stack -- becomes the current entry.  Kernels interleave the
// steps of many rays per warp and refill lanes whose ray has finished.  The
// stack holds one record per tree level on the walk's path; kRecs (from STACK,
// which the host picks from the tree depth) plus kRing records cover every tree
// the host admits.  Should they not, cnt.overflow is set and the result must be
// discarded.
template <int STACK>
struct Traversal {
  float3 lo, hi;
  float t0, t1;
  uint32_t node, octant, hit_ref;   // octant: the ray's in bits 0-2, kSlowSlab, kAnyHit, the entry's gate
  uint32_t lp, lend;         // surface list still to test: plist[lp, lend), lp <= lend
  uint32_t ring;             // shared-memory ring: position of its newest record
  uint32_t held;             // records in the ring
  int sp;                    // older records, in stk[0, sp)
  bool have;                 // a current entry (node, gate, lo, hi) is set
  const uint4 *nodes;        // the ray's scene (its list and primitive arrays are in the ray slot)
  // Records the stack may need: one per tree level.  STACK, the class the
  // host picks from the tree depth (at least 3 * depth + 4), bounds them
  // with room to spare.
  static constexpr int kRecs = (STACK + 2) / 3;
  // The spilled part of the stack: an array of kRecs records owned by the
  // caller.  It is not a member: a dynamically indexed member array puts
  // the whole object in local memory, every scalar above included.
  StackRec *stk;

  // The ray's origin and direction, from its shared-memory slot.
  __device__ __forceinline__ float3 ray_o() const {
    const uint4 a = ray_slots()[threadIdx.x];
    return f3(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z));
  }
  __device__ __forceinline__ float3 ray_d() const {
    const uint4 a = ray_slots()[kTraceBlock + threadIdx.x];
    return f3(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z));
  }
  // Shrink the ray (closest queries), in the register and in the slot.
  __device__ __forceinline__ void set_t1(float t) {
    t1 = t;
    reinterpret_cast<uint32_t *>(ray_slots() + kTraceBlock + threadIdx.x)[3] = __float_as_uint(t);
  }

  __device__ __forceinline__ void init(const DevScene &s, float3 o, float3 d, float t0_, float t1_) {
    t0 = t0_;
    t1 = t1_;
    hit_ref = PREF_END;
    sp = 0;
    ring = 0;
    held = 0;
    node = 0;
    lp = lend = 0;
    have = s.n_nodes != 0;
    nodes = s.nodes;
    {
      uint4 *slot = ray_slots() + threadIdx.x;
      const unsigned long long pl = reinterpret_cast<uintptr_t>(s.lrec);
      slot[0] = make_uint4(__float_as_uint(o.x), __float_as_uint(o.y), __float_as_uint(o.z), __float_as_uint(t0_));
      slot[kTraceBlock] =
          make_uint4(__float_as_uint(d.x), __float_as_uint(d.y), __float_as_uint(d.z), __float_as_uint(t1_));
      reinterpret_cast<uint2 *>(slot + 2 * kTraceBlock)[0] = make_uint2(uint32_t(pl), uint32_t(pl >> 32));
    }
    // 1 / d rounded once, as the reference's division (__frcp_rn is the
    // correctly rounded reciprocal, the same value as 1.0f / d).
    float inv = (d.x == 0.f) ? 1e9f : __frcp_rn(d.x);
    float a = __fmul_rn(__fsub_rn(s.origin[0], o.x), inv);
    float b = __fmul_rn(__fadd_rn(__fsub_rn(s.origin[0], o.x), s.size), inv);
    if (a > b) { float tmp = a; a = b; b = tmp; }
    lo.x = a; hi.x = b;
    inv = (d.y == 0.f) ? 1e9f : __frcp_rn(d.y);
    a = __fmul_rn(__fsub_rn(s.origin[1], o.y), inv);
    b = __fmul_rn(__fadd_rn(__fsub_rn(s.origin[1], o.y), s.size), inv);
    if (a > b) { float tmp = a; a = b; b = tmp; }
    lo.y = a; hi.y = b;
    inv = (d.z == 0.f) ? 1e9f : __frcp_rn(d.z);
    a = __fmul_rn(__fsub_rn(s.origin[2], o.z), inv);
    b = __fmul_rn(__fadd_rn(__fsub_rn(s.origin[2], o.z), s.size), inv);
    if (a > b) { float tmp = a; a = b; b = tmp; }
    lo.z = a; hi.z = b;
    octant = (d.x >= 0.f ? 0u : 4u) | (d.y >= 0.f ? 0u : 2u) | (d.z >= 0.f ? 0u : 1u);
    // A node's bounds lie within its parent's (a far half's upper bound may
    // round one ulp beyond): with every root bound below 1e37 in magnitude
    // no bound below overflows, none is NaN, and with t0, t1 not NaN
    // node_step may take its fast tests.  (fabsf(NaN) < x is false.)
    const bool finite = fabsf(lo.x) < 1e37f && fabsf(lo.y) < 1e37f && fabsf(lo.z) < 1e37f &&
                        fabsf(hi.x) < 1e37f && fabsf(hi.y) < 1e37f && fabsf(hi.z) < 1e37f && !isnan(t0) &&
                        !isnan(t1);
    if (!finite) octant |= kSlowSlab;
  }

  // The walk is over: no list pending, no current entry.
  __device__ __forceinline__ bool finished() const { return lp == lend && !have; }

  // Push a record: into the ring, first moving the ring's oldest record --
  // the one after the newest -- to local memory when the ring is full.
  __device__ __forceinline__ void push(float3 half, uint32_t first, uint32_t bits, TraceCounters &cnt) {
    ring = (ring + 1u) % kRing;
    float4 *r = ring_slots() + 2u * kTraceBlock * ring;
    if (held == kRing) {
      if (sp < kRecs) {
        stk[sp].a = r[0];
        stk[sp].b = r[kTraceBlock];
        sp++;
      } else {
        cnt.overflow = 1;
      }
    } else {
      held++;
    }
    r[0] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(first));
    r[kTraceBlock] = make_float4(half.x, half.y, half.z, __uint_as_float(bits));
  }

  // One octree entry (call only with a current entry and no list pending).
  //
  // An entry is processed as one call of the reference's recursive function:
  // parent gate, slab cull, then the node's surface list, then its children.
  // Here the qualifying children are pushed when the node is visited and its
  // list is tested afterwards; the push uses the ray's extent before those
  // tests, which only admits more children (the ray can only shrink), and a
  // closest-hit query's entries are culled again when they are entered -- so
  // the tests and their order are the reference's.
  // ANY: the queries the calling kernel runs -- kClosestOnly, kAnyOnly or
  // kMixed (checked per ray) -- so closest-hit kernels carry no any-hit branch.
  // COUNT: node calls are counted.
  template <int ANY, bool COUNT>
  __device__ __forceinline__ void node_step(TraceCounters &cnt) {
    const bool slow = octant & kSlowSlab;
    bool open = true;
    const bool any_query = ANY == kAnyOnly || (ANY == kMixed && (octant & kAnyHit));
    if (ANY == kAnyOnly || ((octant & kGateFlag) && any_query)) {
      // An any-hit query's extent never changes, so an entry with a parent
      // gate passed the very gate and cull it would be given now when it
      // was pushed (or entered): the call happens and the node is open.
      // (The root of an any-hit kernel's rays passed its cull at the start.)
      if (COUNT) cnt.nodes++;
    } else {
      // The cull decides alone where bounds are finite: it closes whatever the
      // gate does.  The gate is where a call is counted.
      if ((COUNT || slow) && (octant & kGateFlag)) open = gate_open(octant >> kGateShift, t0, t1, lo, hi);
      if (open) {
        if (COUNT) cnt.nodes++;
        open = slow ? slab_open(t0, t1, lo, hi) : slab_open_finite(t0, t1, lo, hi);
      }
    }
    // The record whose children come next: the node's own if any of them
    // qualifies, else the newest on the stack.
    float3 half = lo;
    uint32_t first = 0, bits = 0, vm = 0;   // bits: child mask, children of a stacked record still to enter << 8
    if (open) {
      const uint4 nd = __ldg(nodes + node);
      lp = nd.z;
      lend = nd.z + nd.w;
      first = nd.x;
      bits = nd.y & 0xffu;
      if (nd.y) {
        // (hi - lo) / 2: halving rounds exactly like the reference's division by 2.
        half = f3(__fmul_rn(__fsub_rn(hi.x, lo.x), 0.5f), __fmul_rn(__fsub_rn(hi.y, lo.y), 0.5f),
                  __fmul_rn(__fsub_rn(hi.z, lo.z), 0.5f));
        // Per axis the children's bounds take two values each: the near half
        // spans [lo, lo + half], the far half [lo + half, lo + half + half] --
        // the same rounded sums as the reference's child ranges.
        const float3 mid = f3(__fadd_rn(lo.x, half.x), __fadd_rn(lo.y, half.y), __fadd_rn(lo.z, half.z));
        const float3 far = f3(__fadd_rn(mid.x, half.x), __fadd_rn(mid.y, half.y), __fadd_rn(mid.z, half.z));
        // Which children pass gate and cull, by octant bits.  At most 4 pass: one
        // octant per crossing of each of the three midplanes.
        const uint32_t oct = octant & 7u;
        if (slow) {
#pragma unroll
          for (uint32_t cb = 0; cb < 8; cb++) {
            const float3 clo = f3((cb & 4) ? mid.x : lo.x, (cb & 2) ? mid.y : lo.y, (cb & 1) ? mid.z : lo.z);
            const float3 chi = f3((cb & 4) ? far.x : mid.x, (cb & 2) ? far.y : mid.y, (cb & 1) ? far.z : mid.z);
            const bool ok =
                ((nd.y >> (cb ^ oct)) & 1u) & gate_open(cb, t0, t1, clo, chi) & slab_open(t0, t1, clo, chi);
            vm |= ok ? (1u << cb) : 0u;
          }
        } else {
          // The same tests taken apart.  lo <= mid <= far per axis (half is not
          // negative where the node is open), so a child's entry is the largest
          // of ENTRY and the midpoints of its far axes, its exit the smallest of
          // EXIT and the midpoints of its near axes, and entry < exit holds
          // exactly when each of the former is below each of the latter: a far
          // axis' midpoint below EXIT, a near one's above ENTRY, and a far axis'
          // midpoint below a near one's.  Each failed comparison takes its
          // children out of the mask.  The gates follow from the same
          // comparisons.  (Against a maximum, a minimum and four gates for each of
          // eight children: terrain frame 224.5 -> 201.8 ms, 16M rays in 1M
          // triangles 20.2 -> 17.6 ms, with the uncounted cull above.)
          const float entry = fmaxf(fmaxf(t0, lo.x), fmaxf(lo.y, lo.z));
          const float exit = fminf(fminf(t1, far.x), fminf(far.y, far.z));
          vm = (__byte_perm(nd.y, 0u, (oct & 3u) * 0x1111u) >> (oct & 4u)) & 0xffu;   // children that exist
          if (!(entry < exit)) vm = 0u;
          if (!(entry < mid.x)) vm &= 0xf0u;
          if (!(entry < mid.y)) vm &= 0xccu;
          if (!(entry < mid.z)) vm &= 0xaau;
          if (!(mid.x < exit)) vm &= 0x0fu;
          if (!(mid.y < exit)) vm &= 0x33u;
          if (!(mid.z < exit)) vm &= 0x55u;
          if (!(mid.x < mid.y)) vm &= ~0x30u;   // x far, y near
          if (!(mid.y < mid.x)) vm &= ~0x0cu;
          if (!(mid.x < mid.z)) vm &= ~0x50u;   // x far, z near
          if (!(mid.z < mid.x)) vm &= ~0x0au;
          if (!(mid.y < mid.z)) vm &= ~0x44u;   // y far, z near
          if (!(mid.z < mid.y)) vm &= ~0x22u;
        }
      }
    }
    // The first qualifying child becomes the current entry; the others wait
    // in one record and are entered in visiting order after the first
    // child's subtree, as the reference's loop over the children does.
    const bool popped = vm == 0u;
    if (popped) {
      float4 ra, rb;
      if (held) {
        const float4 *r = ring_slots() + 2u * kTraceBlock * ring;
        ra = r[0];
        rb = r[kTraceBlock];
      } else if (sp) {
        ra = stk[sp - 1].a;
        rb = stk[sp - 1].b;
      } else {
        have = false;
        return;
      }
      lo = xyz(ra);
      half = xyz(rb);
      first = __float_as_uint(ra.w);
      bits = __float_as_uint(rb.w);
      vm = bits >> 8;
    }
    const uint32_t cb = first_child(vm);
    const uint32_t rest = vm & ~(1u << cb);
    const uint32_t word = (bits & 0xffu) | (rest << 8);
    if (!popped) {
      if (rest) push(half, first, word, cnt);
    } else if (held) {
      if (rest) {
        reinterpret_cast<uint32_t *>(ring_slots() + (2u * ring + 1u) * kTraceBlock)[3] = word;
      } else {
        held--;
        ring = (ring + kRing - 1u) % kRing;
      }
    } else if (rest) {
      stk[sp - 1].b.w = __uint_as_float(word);
    } else {
      sp--;
    }
    node = first + __popc(bits & ((1u << (cb ^ (octant & 7u))) - 1u));
    if (COUNT || slow) octant = (octant & (kGateFlag - 1u)) | kGateFlag | (cb << kGateShift);
    else if (ANY == kMixed) octant |= kGateFlag;
    // The far half starts at mid; either half ends half an extent after it starts.
    if (cb & 4) lo.x = __fadd_rn(lo.x, half.x);
    if (cb & 2) lo.y = __fadd_rn(lo.y, half.y);
    if (cb & 1) lo.z = __fadd_rn(lo.z, half.z);
    hi = f3(__fadd_rn(lo.x, half.x), __fadd_rn(lo.y, half.y), __fadd_rn(lo.z, half.z));
  }
};

// One warp-cooperative round of list tests.  Every lane with a list pending
// owns the next entries of its list; the warp's pending entries, in
// lane order and list order, are dealt to its 32 lanes (one or two
// consecutive entries per lane: at most 32 or 64 per round), each lane tests
// its entries against its owner's ray, and each owner takes the result of its
// own entries:
//  * closest queries: the smallest hit t, the earliest entry among equal t.
//    This is what the sequential test with a shrinking t1 keeps -- an entry
//    hits when its t (which does not depend on t1) is below t1 -- so the
//    result equals the reference's one-by-one loop;
//  * any-hit queries (ANY): the earliest entry that hits, where the
//    reference's loop stops.
// Test counts are the reference's (all entries, or up to the stopping one).
// All 32 lanes must call it together.  Returns true for an any-hit lane whose
// search is over.
// PER: entries dealt to a lane per round, 1 or 2.  Pairs (two consecutive
// entries of one list per lane, up to 64 per round) pay where the lists a
// ray meets are long and the warps have rays to fill the rounds: the
// closest-hit kernels use them for scenes whose probe found long lists along
// rays (SceneImpl's pair_lists: a 2M-triangle soup render 13.1 -> 12.1 ms, a
// 50k-triangle one, whose lists are short, 6.2 -> 6.8), the ray-batch kernel for
// those scenes and batches that fill the device (trace.cu).  Any-hit rounds
// deal single entries: a walk stops at its first hit (pairs: shadow rays of the
// terrain frame 50.6 -> 57.3 ms, of a 200k-triangle soup 4.9 -> 5.5).
//
// Bookkeeping.  An owner's units are consecutive lanes [excl, excl + np), so
// one ballot of the hits gives every owner its own hits by a mask; the few
// that hit are compared in a loop over each owner's hits (most often none or
// one).  The k-th owner leaves what its units need in the warp's k-th ray
// slot, where a unit finds it by counting the first units at or before its
// lane.  (Against a match over the owners, two reductions per owner's group
// and a five-shuffle search per unit: terrain frame 273.3 -> 225.5 ms, 16M
// rays in 1M triangles 24.7 -> 20.15 ms.)
template <int STACK, int ANY, int PER>
__device__ __forceinline__ bool list_round(Traversal<STACK> &tr, bool any, TraceCounters &cnt) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr uint32_t kPer = uint32_t(PER);
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t c = tr.lend - tr.lp;
  c = c < 32u * kPer ? c : 32u * kPer;
  const uint32_t np = (c + kPer - 1u) / kPer;   // dealt units: pairs (or entries)
  uint32_t incl = np;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    // incl += its value OFF lanes below, where there is such a lane (the shuffle's own predicate says).
    asm volatile(
        "{\n .reg .pred p;\n .reg .u32 v;\n shfl.sync.up.b32 v|p, %0, %1, 0, 0xffffffff;\n @p add.u32 %0, %0, v;\n}"
        : "+r"(incl)
        : "r"(off));
  }
  const uint32_t excl = incl - np;
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0u) return false;
  const bool owner = np > 0u && excl < 32u;
  const uint32_t owners = __ballot_sync(kFull, owner);
  const uint32_t starts = __reduce_or_sync(kFull, owner ? (1u << excl) : 0u);
  uint4 *const wslot = ray_slots() + (threadIdx.x & ~31u);
  if (owner) {
    // First entry of a unit at lane l: base + kPer * l; entries end at base + stop.
    const uint32_t k = __popc(owners & ((1u << lane) - 1u));
    reinterpret_cast<uint2 *>(wslot + 2 * kTraceBlock + k)[1] =
        make_uint2(tr.lp - kPer * excl, lane | (any ? 32u : 0u) | ((kPer * excl + c) << 8));
  }
  __syncwarp();   // these, and the warp's ray-slot writes (new rays, shrunk t1), are visible
  uint32_t pid = PREF_END, which = 0u;
  bool hit = false;
  float th = 0.f;
  if (lane < total) {
    const uint32_t k = __popc(starts & (kFull >> (31u - lane))) - 1u;
    const uint2 unit = reinterpret_cast<const uint2 *>(wslot + 2 * kTraceBlock + k)[1];
    const uint4 *slot = wslot + (unit.y & 31u);
    const uint4 ra = slot[0], rb = slot[kTraceBlock];
    const uint2 rc = reinterpret_cast<const uint2 *>(slot + 2 * kTraceBlock)[0];
    const float3 ro = f3(__uint_as_float(ra.x), __uint_as_float(ra.y), __uint_as_float(ra.z));
    const float3 rd = f3(__uint_as_float(rb.x), __uint_as_float(rb.y), __uint_as_float(rb.z));
    const float rt0 = __uint_as_float(ra.w);
    const float rt1 = __uint_as_float(rb.w);
    // The entries' primitive records from the owner's scene's list records.
    const unsigned long long o_lrec = (unsigned long long)rc.x | ((unsigned long long)rc.y << 32);
    const float4 *p = reinterpret_cast<const float4 *>(o_lrec) + 3 * size_t(unit.x + kPer * lane);
    const PrimRec r0{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
    th = rt1;
    hit = test_prim(r0, ro, rd, rt0, th);
    pid = __float_as_uint(r0.c.w);
    if (kPer == 2u && kPer * lane + 1u < (unit.y >> 8) && !(ANY != kClosestOnly && hit && (unit.y & 32u))) {
      const PrimRec r1{__ldg(p + 3), __ldg(p + 4), __ldg(p + 5)};
      float th1 = rt1;
      const bool hit1 = test_prim(r1, ro, rd, rt0, th1);
      // The later entry wins only with a smaller t (the earlier one keeps ties).
      if (hit1 && (!hit || th1 < th)) {
        hit = true;
        th = th1;
        pid = __float_as_uint(r1.c.w);
        which = 1u;
      }
    }
  }
  const uint32_t hits = __ballot_sync(kFull, hit);
  const uint32_t room = 32u - excl;   // (excl > 31 only where !owner)
  uint32_t mine = owner ? hits & ((np < room ? (1u << np) - 1u : kFull) << excl) : 0u;
  bool over = false;
  if (hits) {   // the same for the whole warp
    const bool found = mine != 0u;
    uint32_t best = found ? uint32_t(__ffs(mine)) - 1u : lane;
    float b_t = __shfl_sync(kFull, th, best);
    if (ANY != kAnyOnly) {
      if (ANY == kMixed && any) mine = 0u;   // the earliest stands
      mine &= mine - 1u;
      while (__any_sync(kFull, mine != 0u)) {
        const uint32_t src = mine ? uint32_t(__ffs(mine)) - 1u : lane;
        const float t = __shfl_sync(kFull, th, src);
        if (mine && t < b_t) {
          b_t = t;
          best = src;
        }
        mine &= mine - 1u;
      }
    }
    const uint32_t b_pid = __shfl_sync(kFull, pid, best);
    const uint32_t b_which = kPer == 2u && ANY != kClosestOnly ? __shfl_sync(kFull, which, best) : 0u;
    if (found) {
      tr.hit_ref = b_pid;
      if (ANY != kClosestOnly && any) {
        cnt.tests += kPer * (best - excl) + b_which + 1u;
        tr.lp = tr.lend;
        over = true;
      } else {
        tr.set_t1(b_t);
      }
    }
  }
  if (owner && !over) {
    const uint32_t used = c < kPer * room ? c : kPer * room;
    cnt.tests += used;
    tr.lp += used;
  }
  return over;
}

// Idle lanes a warp gathers before it refills them (1 = refill at once): 8 in
// the renderers' kernels, 4 in the ray-batch kernel, whose ray starts read
// less (terrain frame 193.0 ms at 4, 190.9 at 8; 1M rays among 22k mixed
// primitives 0.82 ms at 4, 0.86 at 8).
#ifndef SNOG_REFILL_MIN
#define SNOG_REFILL_MIN 8
#endif
constexpr uint32_t refill_min(int any) { return any == kMixed ? 4u : uint32_t(SNOG_REFILL_MIN); }

// Pending list entries a closest-hit warp gathers before a list round, and
// the lanes able to visit a node below which it does not wait for more
// (closest-hit kernel of the terrain frame 77.2 ms at 24 and 0, 76.3 at 16
// and 4).
#ifndef SNOG_ROUND_MIN
#define SNOG_ROUND_MIN 16
#endif
constexpr uint32_t kRoundMin = SNOG_ROUND_MIN;
constexpr uint32_t kFewSteps = 4;
// A warp with fewer than 32 entries pending visits nodes, and one with at
// least kRoundMin, or no lane that could visit one, runs a round; a threshold
// above 32 would leave a warp with 32..kRoundMin-1 entries pending doing
// neither, for ever.
static_assert(kRoundMin >= 1u && kRoundMin <= 32u, "closest-hit round threshold must not exceed the node-step cut");

// Warp-cooperative ray dispenser for the persistent trace kernels: lanes
// whose ray is finished take the next index from a warp-local range of up to
// 32 rays.  A warp's first range is its own place in the launch, later ones
// take one atomic on the launch's counter: a launch with fewer rays than lanes
// needs none (thousands of warps adding to one address take microseconds).
// All 32 lanes of the warp must call fetch() together.
//
// A launch lasts as long as its slowest warp, and a warp with few rays runs
// through their lists faster than one with 32 (its list rounds are shared by
// fewer rays).  So a launch with fewer rays than lanes spreads them: each warp
// holds at most its even share, LIMIT of 1 to 32 rays, in its first LIMIT
// lanes.  999 rays among 10k triangles 147 -> 99 us, a 64x48 Cornell render
// 803 -> 621 us, the late bounces of an 853x479 terrain render 12.5 -> 11.6
// ms; launches with 32 rays a warp are unchanged (ranges that shrink with the
// rays left, besides, measured 1-2 % slower there).  The own first ranges: the
// same small batch 87 -> 82 us, the small Cornell render 598 -> 552 us.
struct RayDispenser {
  static constexpr uint32_t kIdle = 0xffffffffu;
  uint32_t next, end;
  uint32_t limit;   // 0: no rays remain to be handed out

  __device__ __forceinline__ explicit RayDispenser(uint32_t n) {
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t share = n / warps + (n % warps ? 1u : 0u);
    limit = share < 32u ? share : 32u;   // (0 for an empty launch)
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    next = warp * limit < n ? warp * limit : n;
    end = limit < n - next ? next + limit : n;
  }

  // The new ray index for a lane that asked (NEED) and got one, else kIdle.
  __device__ __forceinline__ uint32_t fetch(uint32_t *counter, uint32_t n, bool need) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t mask = __ballot_sync(0xffffffffu, need);
    if (next == end) {
      const uint32_t first = gridDim.x * (blockDim.x >> 5) * limit;   // rays in the warps' own ranges
      uint32_t base = n;
      if (lane == 0 && first < n) base = atomicAdd(counter, limit);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (first >= n || base >= n - first) {
        limit = 0;
      } else {
        next = first + base;
        end = n - next < limit ? n : next + limit;
      }
    }
    const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
    const uint32_t got = need && rank < end - next ? next + rank : kIdle;
    const uint32_t take = __popc(mask);
    next = take < end - next ? next + take : end;
    return got;
  }
};

// The persistent trace loop shared by the trace kernels.  Lanes take rays
// from DISPENSER (n rays) through a RayDispenser; START(i, tr, any) begins ray
// i (calls tr.init and sets ANY for an any-hit query); DONE(i, tr, any)
// stores its result.  Each iteration, unless the warp already has a full
// round of list entries pending, every live lane without a list pending
// visits one octree entry; then the warp tests one round of pending list
// entries together.  All 32 lanes of every warp must run it.
//
// The loop is bound by instructions issued: on the terrain frame the
// closest-hit kernel runs 0.86 node steps (25.8 lanes on average), 0.76 list
// rounds (31.1 entries) and 0.24 refills an iteration, so what counts is
// the length of each.  Against popping the next entry at the start of a step,
// a third 16-byte part per stack record and a vote on every refill, with
// the ring of 4 records that the smaller ones make room for: terrain frame
// 201.9 -> 190.9 ms, 16M rays in 1M triangles 17.6 -> 16.4 ms, 200k-triangle
// soup 19.8 -> 17.7 ms.  One reduction for pending entries and waiting lanes,
// the refill threshold in a register, the scan's additions under the shuffle's
// own predicate, no gate word and no entry test where a kernel does not
// need them: terrain frame 170.0 -> 167.0 ms.
template <int STACK, int ANY, int PER, bool COUNT, class Start, class Done>
__device__ __forceinline__ void trace_loop(uint32_t *dispenser, uint32_t n, TraceCounters &cnt, Start start,
                                           Done done) {
  StackRec stk[Traversal<STACK>::kRecs];
  Traversal<STACK> tr;
  tr.stk = stk;
  RayDispenser disp(n);
  tr.have = false;
  tr.lp = tr.lend = 0;
  uint32_t ray = RayDispenser::kIdle;
  bool any = false;
  // Idle lanes take new rays only once refill_min of those that may are idle:
  // a ray start (queue loads, root slab set-up, ray slot) then runs on several
  // lanes at once instead of on one or two every iteration.
  // (The ray-batch kernel has no register for the threshold: 16M rays 15.7 ms
  // without, 16.4 with.)
  uint32_t refill_at = 32u - disp.limit + (refill_min(ANY) < disp.limit ? refill_min(ANY) : disp.limit);
  for (;;) {
    const uint32_t idle = __ballot_sync(0xffffffffu, ray == RayDispenser::kIdle);
    if (ANY == kMixed)
      refill_at = disp.limit ? 32u - disp.limit + (refill_min(ANY) < disp.limit ? refill_min(ANY) : disp.limit) : 33u;
    if (uint32_t(__popc(idle)) >= refill_at) {
      const uint32_t got =
          disp.fetch(dispenser, n, ray == RayDispenser::kIdle && (threadIdx.x & 31u) < disp.limit);
      if (disp.limit == 0u) refill_at = 33u;   // never again
      if (got != RayDispenser::kIdle) {
        ray = got;
        start(ray, tr, any);
        if (any) tr.octant |= kAnyHit;
        if (ANY == kAnyOnly && tr.have && !slab_open(tr.t0, tr.t1, tr.lo, tr.hi)) {
          if (COUNT) cnt.nodes++;
          tr.have = false;
        }
      }
    } else if (idle == 0xffffffffu) {
      break;
    }
    // Visit nodes only while the warp's pending list entries would not fill
    // a round: list rounds run full, node steps run with more lanes at once.
    const uint32_t pend = tr.lend - tr.lp;
    const uint32_t pending = __reduce_add_sync(0xffffffffu, pend < 32u ? pend : 32u);
    if (pending < 32u && tr.have && pend == 0u) tr.template node_step<ANY, COUNT>(cnt);
    // Closest-hit kernels test lists only once at least kRoundMin entries are
    // pending or few lanes could visit a node: fewer, fuller rounds.  (Any-hit
    // and mixed kernels, whose walks end early or whose lists are longer,
    // measured a loss: shadow rays of the terrain frame 60.5 -> 62.5 ms.)
    bool round = true;
    if (ANY == kClosestOnly) {
      const uint32_t pend2 = tr.lend - tr.lp;
      // Pending entries (at most 1024) and, above them, lanes that could visit a node.
      const uint32_t both = __reduce_add_sync(
          0xffffffffu, pend2 ? (pend2 < 32u ? pend2 : 32u) : tr.have ? 1u << 16 : 0u);
      round = (both & 0xffffu) >= kRoundMin || both < (kFewSteps + 1u) << 16;
    }
    const bool stop = round && list_round<STACK, ANY, PER>(tr, any, cnt);
    if (ray != RayDispenser::kIdle && (stop || tr.finished())) {
      done(ray, tr, any);
      tr.have = false;
      ray = RayDispenser::kIdle;
    }
  }
}

// Global primitive id of a packed reference: triangles, then spheres, then
// tripars.
__device__ __forceinline__ int32_t prim_id_of(const DevScene &, uint32_t ref) {
  return ref == PREF_END ? -1 : int32_t(ref);
}

}  // namespace snog

#endif
