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

// ray_box with the result in one word: the child's entry distance, or NaN
// when it is not to be entered, i.e. unless ray_box(..., bt, tn) && tn <= bt.
// The exit is widened before it is clamped by bt, which is the same test:
// entry <= min(exit, bt) x kBoxHi and entry <= bt hold together exactly when
// entry <= min(exit x kBoxHi, bt), bt being no less than zero.
__device__ __forceinline__ float child_entry(const ChildPairs &n, const RayPairs &r, float bt) {
  float x0, y0, z0, x1, y1, z1;
  up2(mul2_rn(add2_rn(n.b[0], r.nxy), r.ixy), x0, y0);
  up2(mul2_rn(add2_rn(n.b[1], r.nxy), r.ixy), x1, y1);
  up2(mul2_rn(add2_rn(n.b[2], r.nzz), r.izz), z0, z1);
  const float tn =
      __fmul_rn(fmaxf(max3f(nan_min(x0, x1), nan_min(y0, y1), nan_min(z0, z1)), r.tmin), kBoxLo);
  const float tf = __fmul_rn(min3f(nan_max(x0, x1), nan_max(y0, y1), nan_max(z0, z1)), kBoxHi);
  return tn <= fminf(tf, bt) ? tn : __int_as_float(0x7fffffff);
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
    t = top_t = 0.0f;
    sp = 0;
  }
};
// Moves on: t0, t1 are the entry distances of the children (NaN: not to be
// entered) of the lane's node, on whether it has one.  Returns false when the
// stack is full.
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
// every warp that fits on the GPU; fewer rays are spread over the warps
// instead, at least four to each (a warp's time is that of its longest ray,
// and lanes without a ray still run queued primitive tests).  4,099 rays on
// 1,501 triangles at 32 / 16 / 8 / 4 / 2 / 1 rays per warp: 102 / 85 / 81 /
// 78 / 78 / 93 us.
struct RayGrid {
  int ctas, lanes;
};
static inline RayGrid ray_grid(uint64_t nrays, int ctas, int warps) {
  const uint64_t fit = (uint64_t)gprtcu_num_sms() * ctas;
  const uint64_t share = (nrays + fit * warps - 1) / (fit * warps);
  const int lanes = share >= 32 ? 32 : (share < 4 ? 4 : (int)share);
  const uint64_t need = (nrays + (uint64_t)lanes * warps - 1) / ((uint64_t)lanes * warps);
  return RayGrid{(int)(need < fit ? need : fit), lanes};
}
