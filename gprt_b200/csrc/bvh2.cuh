// bvh2.cuh -- one step of a binary-LBVH traversal, shared by the ray kernels:
// the node fetch, the test of its two child boxes, and the traversal stack.
#pragma once
#include "common.cuh"
#include "lbvh.cuh"
#include "rtmath.cuh"

namespace gprtcu {

// A child's box in pairs, in memory order: (lo.x, lo.y), (hi.x, hi.y),
// (lo.z, hi.z); and its reference.
struct ChildPairs {
  unsigned long long b[3];
  int ref;
};

// Half a node, one child.  Lanes visit different nodes, so a warp's load costs
// L1 one cycle per lane and instruction however wide it is, and that is what
// bounds the triangle walk: with four 16-byte loads per node the L1 data pipe
// was 87 % busy at 12 of 32 lanes active (1,048,576 rays on 262,144
// triangles, 2.65 ms); two 32-byte loads alone gave 2.32 ms.  They need nodes
// on 32-byte boundaries; V8 = false serves arrays that are only 16-byte
// aligned.  (Measured and not kept: the two lanes of a pair fetching half of
// each other's nodes, so a pair's loads fall into one line: L1 at 49 %, but
// both rays in each lane's registers leave 24 warps per SM, 2.30 ms; one ray
// per pair of lanes: 16 rays per warp take 1.9 G instead of 1.1 G warp
// instructions, 2.28 ms.)
template <bool V8> __device__ __forceinline__ ChildPairs load_child(const Bvh2Child *p) {
  ChildPairs n;
  unsigned long long rf;
  if constexpr (V8) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(n.b[0]), "=l"(n.b[1]), "=l"(n.b[2]), "=l"(rf)
        : "l"(p));
  } else {
    asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(n.b[0]), "=l"(n.b[1]) : "l"(p));
    asm("ld.global.nc.v2.b64 {%0, %1}, [%2];"
        : "=l"(n.b[2]), "=l"(rf)
        : "l"(reinterpret_cast<const char *>(p) + 16));
  }
  n.ref = (int)(uint32_t)rf;
  return n;
}

// A ray's origin (negated) and reciprocal direction in the pairs that a box's
// words come in, so its slab distances are three packed subtractions and
// three packed products (each half rounds as the scalar operation of ray_box
// does, so the distances have the same bits).
struct RayPairs {
  unsigned long long nxy, nzz, ixy, izz;
  float tmin;
};
__device__ __forceinline__ RayPairs ray_pairs(const Ray &r) {
  return RayPairs{pk2(-r.ox, -r.oy), pk2(-r.oz, -r.oz), pk2(r.ix, r.iy), pk2(r.iz, r.iz), r.tmin};
}

// ray_box(..., bt, tn) && tn <= bt of a child's box, bt being a number.
// The exit is widened before it is clamped by bt, which is the same test:
// entry <= min(exit, bt) x kBoxHi and entry <= bt hold together exactly when
// entry <= min(exit x kBoxHi, bt), bt being no less than zero.
__device__ __forceinline__ bool child_hit(const ChildPairs &n, const RayPairs &r, float bt, float &tn) {
  float x0, y0, z0, x1, y1, z1;
  up2(mul2_rn(add2_rn(n.b[0], r.nxy), r.ixy), x0, y0);
  up2(mul2_rn(add2_rn(n.b[1], r.nxy), r.ixy), x1, y1);
  up2(mul2_rn(add2_rn(n.b[2], r.nzz), r.izz), z0, z1);
  tn = __fmul_rn(fmaxf(max3f(nan_min(x0, x1), nan_min(y0, y1), nan_min(z0, z1)), r.tmin), kBoxLo);
  const float tf = __fmul_rn(min3f(nan_max(x0, x1), nan_max(y0, y1), nan_max(z0, z1)), kBoxHi);
  return tn <= fminf(tf, bt);
}
// The same in one word: the child's entry distance, or NaN when it is not to
// be entered.
__device__ __forceinline__ float child_entry(const ChildPairs &n, const RayPairs &r, float bt) {
  float tn;
  return child_hit(n, r, bt, tn) ? tn : __int_as_float(0x7fffffff);
}

// A lane's walk over the tree: its node (negative: the walk is over) with the
// node's entry distance, and a stack whose top entry is kept in registers, so
// a step's push is one predicated store and its pop one predicated load.
// Below the top, the first SHARED entries are in shared memory
// (entry-major: a warp's access has no bank conflict whatever depths its lanes
// are at; in local memory every distinct depth is a cache line of its own),
// the rest -- rare -- in local memory.  An entry is a node and its entry
// distance: an entry behind the best hit is dropped without fetching its
// node.  The bottom entry is negative, which ends the walk.
constexpr int kWalkEnd = INT32_MIN;  // the bottom entry
struct Walk {
  int node, top;
  float t, top_t;  // entry distances of node and top
  int sp;          // entries below the top
  __device__ __forceinline__ void start() {
    node = 0;
    top = kWalkEnd;
    t = top_t = -INFINITY;  // the root is visited whatever the ray's range
    sp = 0;
  }
};
// Puts (node, t) on top of the stack; false when it is full.
template <int THREADS, int SHARED, int DEPTH>
__device__ __forceinline__ bool walk_push(Walk &W, float2 *sh, float2 *over, int node, float t) {
  const float2 e = make_float2(__int_as_float(W.top), W.top_t);
  bool ok = true;
  if (W.sp < SHARED) sh[W.sp * THREADS] = e;
  else if (W.sp < DEPTH) over[W.sp - SHARED] = e;
  else ok = false;
  ++W.sp;
  W.top = node;
  W.top_t = t;
  return ok;
}
template <int THREADS, int SHARED>
__device__ __forceinline__ void walk_pop(Walk &W, const float2 *sh, const float2 *over) {
  W.node = W.top;
  W.t = W.top_t;
  --W.sp;
  const float2 e = W.sp < SHARED ? sh[max(W.sp, 0) * THREADS] : over[W.sp - SHARED];
  W.top = W.sp < 0 ? kWalkEnd : __float_as_int(e.x);
  W.top_t = e.y;
}
// Moves on: t0, t1 are the entry distances of the children (NaN: not to be
// entered) of the lane's node, on whether it has one; a lane without one
// passes NaN twice.  Returns false when the stack is full: the walk is then
// over, and the caller sets W.node to the end.
template <int THREADS, int SHARED, int DEPTH>
__device__ __forceinline__ bool walk_next(Walk &W, float2 *sh, float2 *over, bool on, float t0, int r0, float t1,
                                          int r1) {
  const bool in0 = t0 == t0, in1 = t1 == t1;
  const bool first = in0 && !(t1 < t0);  // the nearer child, child 0 on ties
  bool ok = true;
  if (in0 && in1) ok = walk_push<THREADS, SHARED, DEPTH>(W, sh, over, first ? r1 : r0, fmaxf(t0, t1));
  if (in0 || in1) {
    W.node = first ? r0 : r1;
    W.t = first ? t0 : t1;
  }
  if (on && !in0 && !in1) walk_pop<THREADS, SHARED>(W, sh, over);
  return ok;
}

// ---------------------------------------------------------------------------
// few rays
// ---------------------------------------------------------------------------
// Closest hit of few rays: a warp takes up to kPoolRays rays and all its lanes
// work on them.  With a lane per ray the time of a small call is the chain of
// its longest ray's node visits, a load and some 250 cycles of arithmetic each
// (4,099 rays on 1,501 triangles: 66 us), while most lanes have no ray.  Here
// the nodes still to visit of all the warp's rays are one stack in shared
// memory, (node, ray, entry distance); every step each lane takes one of its
// top 32 entries, tests both children and pushes those to enter, the nearer
// ones last; leaf children go to a second list whose primitive tests run 32 at
// a time.  A ray's chain is then its depth plus its share of the warp's visits
// divided by 32.  Whole calls, lane per ray / pooled: 4,099 rays on 1,501
// triangles 80 / 30 us, on 262,144 triangles 210 / 38 us; 40,001 rays there
// 348 / 156 us.  With more rays the lane per ray is faster (1,048,576: 1.94 /
// 2.9 ms), since nearer nodes are not strictly first (twice the visits on dense
// primitives) and every step reads its ray from shared memory; from how many
// on depends on what a test costs and how deep the tree is, so the callers
// give the line (pool_grid).  The closest
// (t, id) is the same in any order.  Where boxes overlap so much that nearly
// every child is entered, the stack grows to the lanes times the tree's depth;
// from kPoolWide entries on, fewer lanes go on the fuller it is (an eighth of
// what is left), in the end one, whose walk needs no more than the tree's
// depth on top.
constexpr int kPoolRays = 16;
constexpr int kPoolStack = 456;              // entries; a step pops up to 32 and pushes at most 64
constexpr int kPoolWide = 128;               // up to here all lanes go on
static_assert(kPoolStack - 64 - kPoolWide >= 8 * 32, "all lanes at the line");
constexpr int kPoolLeaves = 96;              // a step queues at most 64
constexpr int kPoolThreads = 64;
constexpr int kPoolWarps = kPoolThreads / 32;
constexpr int kPoolCtas = 12;

struct PoolShared {
  uint2 stack[kPoolStack];  // node, entry distance
  float4 ray[kPoolRays][2];  // {-origin, tmin}, {1 / direction, tmax}
  unsigned long long best[kPoolRays];  // closest (t, id)
  uint32_t base[kPoolRays][2];         // first leaf slot and node of the ray's mesh
  uint32_t leaf[kPoolLeaves];
  uint8_t sray[kPoolStack], lray[kPoolLeaves];
};
__device__ __forceinline__ void pool_ray(PoolShared &S, int ray, const Ray &R, uint32_t base_leaf,
                                         uint32_t base_node) {
  S.ray[ray][0] = make_float4(-R.ox, -R.oy, -R.oz, R.tmin);
  S.ray[ray][1] = make_float4(R.ix, R.iy, R.iz, R.tmax);
  S.best[ray] = ((unsigned long long)t_order(R.tmax) << 32) | kMiss;
  S.base[ray][0] = base_leaf;
  S.base[ray][1] = base_node;
}
// All 32 lanes call; lane i's ray (set by pool_ray) starts at its mesh's root
// (root), or has the single leaf of a mesh without inner nodes to test (one).
// PRIMS: test(slot, ray, {-o, tmin}, {1/d, tmax}, aux) gives the (t, id) key
// of a hit or ~0; won(ray, slot, aux) is called for a hit that became the
// ray's best.  False when the stack was too small for the tree.
template <bool BATCHED, bool V8, class PRIMS>
__device__ __forceinline__ bool pool_walk(PoolShared &S, const Bvh2Node *bvh, bool root, bool one,
                                          const PRIMS &prims) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const float kNone = __int_as_float(0x7fffffff);
  int ns = 0, nl = 0;  // stack entries, queued leaves: the same on every lane
  auto push = [&](bool want, int node, float tn, int ray) {
    const unsigned m = __ballot_sync(FULL_MASK, want);
    if (want) {
      const int k = ns + __popc(m & lt);
      S.stack[k] = make_uint2((uint32_t)node, __float_as_uint(tn));
      S.sray[k] = (uint8_t)ray;
    }
    ns += __popc(m);
  };
  auto queue = [&](bool want, uint32_t slot, int ray) {
    const unsigned m = __ballot_sync(FULL_MASK, want);
    if (want) {
      const int k = nl + __popc(m & lt);
      S.leaf[k] = slot;
      S.lray[k] = (uint8_t)ray;
    }
    nl += __popc(m);
  };
  auto flush = [&]() {  // the last up to 32 queued primitive tests
    const int k = nl < 32 ? nl : 32;
    nl -= k;
    __syncwarp();
    unsigned long long key = ~0ull;
    uint32_t slot = 0;
    int ray = 0;
    float aux = 0.0f;
    if (lane < k) {
      slot = S.leaf[nl + lane];
      ray = S.lray[nl + lane];
      key = prims.test(slot, ray, S.ray[ray][0], S.ray[ray][1], aux);
      if (key != ~0ull) atomicMin(&S.best[ray], key);
    }
    __syncwarp();
    if (key != ~0ull && S.best[ray] == key) prims.won(ray, slot, aux);  // one winner per ray
    __syncwarp();
  };
  __syncwarp();
  push(root, root ? (int)S.base[lane][1] : 0, -INFINITY, lane);
  queue(one, one ? S.base[lane][0] : 0u, lane);
  while (true) {
    __syncwarp();
    if (nl >= 32 || (ns == 0 && nl > 0)) flush();
    if (ns == 0) {
      if (nl == 0) break;
      continue;
    }
    const int k = ns <= kPoolWide ? min(ns, 32) : max(min((kPoolStack - 64 - ns) >> 3, 32), 1);
    if (ns + k > kPoolStack) return false;
    ns -= k;
    int ray = 0, r0 = 0, r1 = 0;
    float t0 = kNone, t1 = kNone;
    bool leaf0 = false, leaf1 = false;
    if (lane < k) {
      const uint2 e = S.stack[ns + lane];
      ray = S.sray[ns + lane];
      const float bt = t_from_order((uint32_t)(S.best[ray] >> 32));
      if (__uint_as_float(e.y) <= bt) {
        const Bvh2Node *nd = bvh + e.x;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        const float4 o = S.ray[ray][0], i = S.ray[ray][1];
        const RayPairs P{pk2(o.x, o.y), pk2(o.z, o.z), pk2(i.x, i.y), pk2(i.z, i.z), o.w};
        t0 = child_entry(c0, P, bt);
        t1 = child_entry(c1, P, bt);
        r0 = c0.ref;
        r1 = c1.ref;
        leaf0 = r0 < 0 && t0 == t0;
        leaf1 = r1 < 0 && t1 == t1;
      }
    }
    __syncwarp();  // the entries are taken before others go over them
    const bool in0 = r0 >= 0 && t0 == t0, in1 = r1 >= 0 && t1 == t1;
    const bool near0 = in0 && !(in1 && t1 < t0);
    const int bn = BATCHED ? (int)S.base[ray][1] : 0;
    const uint32_t bl = BATCHED ? S.base[ray][0] : 0u;
    push(in0 && in1, bn + (near0 ? r1 : r0), near0 ? t1 : t0, ray);
    push(in0 || in1, bn + (near0 ? r0 : r1), near0 ? t0 : t1, ray);
    if (__any_sync(FULL_MASK, leaf0 || leaf1)) {
      while (nl > kPoolLeaves - 64) flush();
      queue(leaf0, bl + (uint32_t)~r0, ray);
      queue(leaf1, bl + (uint32_t)~r1, ray);
    }
  }
  __syncwarp();
  return true;
}

// Idle lanes take new rays from the global counter once `refill` of the
// warp's `lanes` are idle (or all are).  Returns true on the lanes that took
// one, its index in r.  All 32 lanes call.
__device__ __forceinline__ bool warp_take(bool active, bool &drained, int lanes, int refill, uint64_t nrays,
                                          unsigned long long *counter, uint64_t &r) {
  const int lane = threadIdx.x & 31;
  const unsigned idle = __ballot_sync(FULL_MASK, !active && lane < lanes);
  const int n_idle = __popc(idle);
  if (drained || (n_idle < refill && n_idle < lanes)) return false;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(counter, (unsigned long long)n_idle);
  base = __shfl_sync(FULL_MASK, base, 0);
  if (base + n_idle >= nrays) drained = true;
  const uint64_t mine = base + __popc(idle & ((1u << lane) - 1u));
  if (active || lane >= lanes || mine >= nrays) return false;
  r = mine;
  return true;
}

}  // namespace gprtcu

// Grid of a persistent ray kernel (`ctas` CTAs of `warps` warps fit on an SM)
// and the rays a warp holds at a time: all 32 lanes once there are rays for
// `spread_warps` warps per SM; fewer rays are spread over that many warps
// instead, at least four to each (a warp's time is that of its longest ray,
// and lanes without a ray still run queued primitive tests).  4,099 rays on
// 1,501 triangles at 32 / 16 / 8 / 4 / 2 / 1 rays per warp: 102 / 85 / 81 / 78
// / 78 / 93 us.  8 / 12 / 16 / 24 warps per SM: any hit of 25,001 rays on 2,657
// triangles 58.4 / 57.6 / 55.5 / 57.9 us, of 56,001 on 20,001 triangles 130 /
// 130 / 131 / 137 us, of 40,001 on 4.2 M triangles 1,063 / 960 / 917 / 908 us.
// Over instances 8, whose rays have more to share: 20,001 rays over 64
// instances of 4 / 64 / 16 meshes 148 / 84 / 70 us with 8 warps per SM, 152 / 87
// / 72 with 16.
constexpr int kSpreadWarps = 16;
struct RayGrid {
  int ctas, lanes;
};
static inline RayGrid ray_grid(uint64_t nrays, int ctas, int warps, int spread_warps = kSpreadWarps) {
  const uint64_t fit = (uint64_t)gprtcu_num_sms() * ctas;
  const uint64_t spread = (uint64_t)gprtcu_num_sms() * spread_warps;
  const uint64_t share = (nrays + spread - 1) / spread;
  const int lanes = share >= 32 ? 32 : (share < 4 ? 4 : (int)share);
  const uint64_t need = (nrays + (uint64_t)lanes * warps - 1) / ((uint64_t)lanes * warps);
  return RayGrid{(int)(need < fit ? need : fit), lanes};
}
// Grid of a pool kernel and the rays a warp takes at a time (two at least); 0
// rays when there are more than `sixths` sixths of a chunk of kPoolRays for
// every warp that fits.
static inline RayGrid pool_grid(uint64_t nrays, int sixths) {
  const uint64_t fit = (uint64_t)gprtcu_num_sms() * gprtcu::kPoolCtas, warps = fit * gprtcu::kPoolWarps;
  if (6 * nrays > warps * gprtcu::kPoolRays * sixths) return RayGrid{0, 0};
  const uint64_t share = (nrays + warps - 1) / warps;
  const int lanes = share > gprtcu::kPoolRays ? gprtcu::kPoolRays : (share < 2 ? 2 : (int)share);
  const uint64_t need = (nrays + (uint64_t)lanes * gprtcu::kPoolWarps - 1) / ((uint64_t)lanes * gprtcu::kPoolWarps);
  return RayGrid{(int)(need < fit ? need : fit), lanes};
}
