// trace.cu -- closest-hit and any-hit traversal of the binary LBVH.
//
// One lane per ray, rays handed out to persistent warps by an atomic counter
// and lanes refilled as their rays finish (rays differ widely in length).
// Each step loads one 64-byte node holding both child boxes, tests both
// boxes, descends into the nearer inner child and pushes the farther one.  A
// child is entered when its entry distance does not exceed the best hit
// (equal distance still enters, so a tie can be won by a lower primitive id).
// Leaf triangles are stored in leaf order.
#include <type_traits>
#include "bvh2.cuh"
#include "common.cuh"
#include "lbvh.cuh"
#include "rtmath.cuh"

namespace gprtcu {

constexpr int kTraceThreads = 128;
constexpr int kTraceWarps = kTraceThreads / 32;
constexpr int kTraceCtas = 8;     // per SM: 64 registers
constexpr int kStackShared = 8;  // stack entries in shared memory
constexpr int kStackDepth = 64;

// Batched form: rays [ray_off[m], ray_off[m+1]) go to mesh m, whose
// primitives are [tri_off[m], tri_off[m+1]); its traversal nodes start at
// tri_off[m] - m and its leaves at tri_off[m] (mesh-local references are
// offset on the fly).  Hits report mesh-local primitive ids.
struct TraceMeshes {
  const uint32_t *tri_off;
  const uint32_t *ray_off;
  uint32_t meshes;
};

__device__ __forceinline__ uint32_t mesh_of_ray(const TraceMeshes &tm, uint64_t r) {
  uint32_t lo = 0, hi = tm.meshes;  // ray_off[lo] <= r < ray_off[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(tm.ray_off + mid) <= r) lo = mid;
    else hi = mid;
  }
  return lo;
}

struct TraceArgs {
  const Bvh2Node *bvh;
  const float4 *leaf;
  uint32_t n;  // triangles (one mesh)
  TraceMeshes tm;
  const float4 *rays;
  uint64_t nrays;
  int lanes;  // rays a warp holds at a time (1 .. 32)
  Hit *hits;
  unsigned long long *counter;
  uint32_t *err;
};

// The leaf box test of a mesh of one triangle, which has no inner node.
__device__ __forceinline__ bool single_leaf_box(const float4 *leaf, uint32_t slot, const Ray &R) {
  const float4 a = __ldg(leaf + 3 * (size_t)slot), b = __ldg(leaf + 3 * (size_t)slot + 1),
               c = __ldg(leaf + 3 * (size_t)slot + 2);
  float tn;
  return ray_box(R, fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)),
                 fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)), R.tmax, tn) &&
         tn <= R.tmax;
}

// Hits whose distance is still to be refined, per warp: a finished ray's
// index and the leaf slot of its triangle.  32 of them are refined together
// with all lanes busy; a lane refining as its own ray ends would leave the
// rest of the warp waiting for a few hundred instructions.
struct RefineQueue {
  unsigned long long ray[64];
  uint32_t slot[64];
};
__device__ __forceinline__ void refine_queued(const TraceArgs &A, RefineQueue &q, int first, int count) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane < count) {
    const unsigned long long r = q.ray[first + lane];
    const uint32_t slot = q.slot[first + lane];
    const float4 o = __ldg(A.rays + 2 * r), d = __ldg(A.rays + 2 * r + 1);
    Ray R;
    R.ox = o.x; R.oy = o.y; R.oz = o.z;
    R.dx = d.x; R.dy = d.y; R.dz = d.z;
    const float4 a = __ldg(A.leaf + 3 * (size_t)slot), b = __ldg(A.leaf + 3 * (size_t)slot + 1),
                 c = __ldg(A.leaf + 3 * (size_t)slot + 2);
    const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
    Hit h;
    h.prim = __float_as_uint(a.w);
    h.t = refine_t(R, v0, v1, v2);
    A.hits[r] = h;
  }
  __syncwarp();
}

// A warp's lanes with `fin` set have finished ray `r`: misses are stored at
// once, hits queued and refined 32 at a time.  nrq: queued hits, the same on
// every lane.
__device__ __forceinline__ void finish_rays(const TraceArgs &A, RefineQueue &q, int &nrq, bool fin, bool hit,
                                            unsigned long long r, uint32_t slot) {
  const int lane = threadIdx.x & 31;
  if (fin && !hit) {
    Hit h;
    h.prim = kMiss;
    h.t = __int_as_float(0x7f800000);
    A.hits[r] = h;
  }
  const unsigned m = __ballot_sync(FULL_MASK, fin && hit);
  if (!m) return;
  if (fin && hit) {
    const int k = nrq + __popc(m & ((1u << lane) - 1u));
    q.ray[k] = r;
    q.slot[k] = slot;
  }
  nrq += __popc(m);
  if (nrq >= 32) {
    nrq -= 32;
    refine_queued(A, q, nrq, 32);  // the last 32: the rest keeps its place
  }
}

// Idle lanes take new rays (warp_take).  Returns true on the lanes that took
// one; base_leaf and base_node are the first leaf slot and node of the ray's
// mesh and n its triangles.
// Rays beyond the 151,552 that 148 SMs hold at once start as soon as this many
// of a warp's lanes are idle: at 8 / 4 lanes 185,001 rays on 5,001 triangles
// take 160 / 156 us.  The rays of a batch are shorter: 77 M rays over 4,096
// meshes at 4 / 8 / 16 lanes 33.6 / 32.4 / 33.3 ms.
constexpr int kTraceRefill = 4;
constexpr int kBatchRefill = 8;
// One mesh whose nodes and leaves (112 bytes a triangle) pass some 560 MB: a
// node that is not in L2 costs so much more from there on that rays which
// start together are worth more than full lanes, since they meet in the upper
// nodes; most of the lanes, then all, have to be idle first.  Rays per call
// as many as triangles, refill at 8 / 24 / 32: 4.2 M 5.7 / 6.8 / 10.2 ms, 6.0
// M 13.5 / 11.6 / 15.6, 8.4 M 25.5 / 21.2 / 23.2; 4.2 M rays on 16.8 M
// triangles 66 / 56 / 52 ms, on 33.6 M 18.5 / 15.8 / 15.5 (any hit alike).
// The meshes of a batch are small, and a warp's rays are of one or two.
// (An argument instead of a template parameter cost 3 %.)  Calls with fewer
// rays than the GPU holds at once hardly refill and do not mind: 130,001 rays
// on 16.8 M triangles 2.76 ms with 32, 2.72 ms with 4; 400,001 6.45 against
// 7.13 ms.
static inline int trace_refill(uint32_t n) {
  if (n <= 5000000u) return kTraceRefill;
  return n <= 12000000u ? 24 : 32;
}

template <bool BATCHED, int REFILL>
__device__ __forceinline__ bool take_rays(const TraceArgs &A, bool active, bool &drained, uint64_t &r, Ray &R,
                                          uint32_t &n, uint32_t &base_leaf, uint32_t &base_node) {
  if (!warp_take(active, drained, A.lanes, REFILL, A.nrays, A.counter, r)) return false;
  ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
  n = A.n;
  base_leaf = base_node = 0;
  if (BATCHED) {
    const uint32_t m = mesh_of_ray(A.tm, r);
    const uint32_t b = __ldg(A.tm.tri_off + m);
    n = __ldg(A.tm.tri_off + m + 1) - b;
    base_leaf = b;
    base_node = b - m;
  }
  return true;
}

// Any hit: a lane tests the leaf triangles it meets at once, child 0 first,
// and the first step with a hit ends its ray (so the hit is the first of the
// near-first order, however the rays share warps).  Few rays wait for a chain
// of visits, so what a visit costs besides its load counts: votes for new and
// finished rays are taken every kAnySteps visits (at every visit: 2,657
// triangles and 56,001 rays 71.4 us, 4.2 M triangles and 4.0 M rays 16.8 ms;
// now 65.5 us, 15.1 ms), the stack holds nodes alone since nothing is culled
// by distance, and with few rays 16 instead of 8 warps per SM share them
// (ray_grid; 40,001 rays on 4.2 M triangles 1,122 -> 911 us).  1,000,001 rays
// on 100,001 triangles: votes at every / 2nd / 4th / 8th visit 1,564 / 1,553 /
// 1,540 / 1,538 us; then nodes alone on the stack 1,470, every 12th visit 1,464
// us.  10 CTAs per SM spill: 1,547 us.  Stack entries in shared memory 12 / 6 /
// 3: 1,461 / 1,474 / 1,547 us.  One pass over the test for the first leaf of a
// step, whichever child it is: 8,001 rays on 100,001 triangles 168 -> 164 us.
//
// A grid of at most kAnyFewCtas per SM (113,664 rays on 148 SMs) asks for no
// more shared memory than those need (kAnyCarveout per cent of what an SM can
// give), which leaves L1 more: its walks wait for loads.  56,001 / 115,001 rays
// on 2,657 triangles 65.4 -> 60.8 us, 80.7 -> 74 us.  28 / 12 per cent: 62.6 / 73
// us, the latter leaving room for three CTAs.  Above, all 8 are worth more:
// 1,000,001 rays on 735 triangles 240 us, 256 with the carveout.
constexpr int kAnySteps = 12;
constexpr int kAnyCtas = 8;
constexpr int kAnyFewCtas = 6;
constexpr int kAnyCarveout = 20;
constexpr int kAnyShared = 12;  // stack entries in shared memory
template <bool BATCHED, bool V8, int REFILL>
__global__ void __launch_bounds__(kTraceThreads, kAnyCtas) k_trace_any(const TraceArgs A) {
  __shared__ int s_stack[kAnyShared][kTraceThreads];
  __shared__ RefineQueue s_rq[kTraceWarps];
  RefineQueue &rq = s_rq[threadIdx.x >> 5];
  bool active = false, drained = false;
  uint64_t r = 0;
  RayPairs P;
  P.nxy = P.nzz = P.ixy = P.izz = 0;
  P.tmin = 0.0f;
  float Sx = 0.0f, Sy = 0.0f, Sz = 0.0f, tmax = 0.0f;
  int axes = 0;  // kx | ky << 2 | kz << 4
  uint32_t base_leaf = 0, base_node = 0, best = kMiss, best_slot = 0;
  float bt = 0.0f;
  int nrq = 0;
  int node = -1, top = -1, sp = 0;  // the walk: its node, the stack's top entry and the entries below it
  int *const sh = &s_stack[0][threadIdx.x];
  int over[kStackDepth - kAnyShared];
  auto leaf_test = [&](uint32_t slot) {
    Ray Q;
    float nx, ny, nz, unused;
    up2(P.nxy, nx, ny);
    up2(P.nzz, nz, unused);
    Q.ox = -nx;
    Q.oy = -ny;
    Q.oz = -nz;
    Q.tmin = P.tmin;
    Q.tmax = tmax;
    Q.Sx = Sx;
    Q.Sy = Sy;
    Q.Sz = Sz;
    Q.kx = axes & 3;
    Q.ky = (axes >> 2) & 3;
    Q.kz = axes >> 4;
    const float4 a = __ldg(A.leaf + 3 * (size_t)slot), b = __ldg(A.leaf + 3 * (size_t)slot + 1),
                 c = __ldg(A.leaf + 3 * (size_t)slot + 2);
    const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
    const uint32_t id = __float_as_uint(a.w);
    float t;
    if (isect_tri(Q, v0, v1, v2, t) && (best == kMiss || t < bt || (t == bt && id < best))) {
      best = id;
      best_slot = slot;
      bt = t;
    }
  };
  while (true) {
    uint32_t n;
    Ray R;
    if (take_rays<BATCHED, REFILL>(A, active, drained, r, R, n, base_leaf, base_node)) {
      active = true;
      best = kMiss;
      P = ray_pairs(R);
      Sx = R.Sx;
      Sy = R.Sy;
      Sz = R.Sz;
      axes = R.kx | (R.ky << 2) | (R.kz << 4);
      bt = tmax = R.tmax;
      node = bt == bt ? 0 : -1;  // no box lies in a range that ends in NaN
      top = -1;
      sp = 0;
      if (n == 1) {
        if (single_leaf_box(A.leaf, base_leaf, R)) leaf_test(base_leaf);
        node = -1;
      }
    }
    if (!__any_sync(FULL_MASK, active)) {
      if (drained) break;
      continue;
    }
#pragma unroll 1
    for (int step = 0; step < kAnySteps; ++step) {
      if (node >= 0) {
        const Bvh2Node *nd = A.bvh + base_node + node;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        float t0, t1;
        const bool h0 = child_hit(c0, P, bt, t0), h1 = child_hit(c1, P, bt, t1);
        const bool l0 = h0 && c0.ref < 0, l1 = h1 && c1.ref < 0;
        if (l0 || l1) {  // a lane's first leaf shares one pass over the test, whichever child it is
          leaf_test(base_leaf + (uint32_t)~(l0 ? c0.ref : c1.ref));
          if (l0 && l1 && t1 <= bt) leaf_test(base_leaf + (uint32_t)~c1.ref);
        }
        const bool in0 = h0 && c0.ref >= 0, in1 = h1 && c1.ref >= 0;
        const bool first = in0 && !(in1 && t1 < t0);  // the nearer child, child 0 on ties
        if (best != kMiss) {
          node = -1;
        } else if (in0 || in1) {
          if (in0 && in1) {
            if (sp < kAnyShared) sh[sp * kTraceThreads] = top;
            else if (sp < kStackDepth) over[sp - kAnyShared] = top;
            ++sp;
            top = first ? c1.ref : c0.ref;
          }
          node = first ? c0.ref : c1.ref;
          if (sp > kStackDepth) {
            atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
            node = -1;
          }
        } else {
          node = top;
          --sp;
          top = sp < 0 ? -1 : (sp < kAnyShared ? sh[sp * kTraceThreads] : over[sp - kAnyShared]);
        }
      }
    }
    const bool fin = active && node < 0;
    if (__any_sync(FULL_MASK, fin)) {
      finish_rays(A, rq, nrq, fin, best != kMiss, r, best_slot);
      if (fin) active = false;
    }
  }
  refine_queued(A, rq, 0, nrq);
}

// Closest hit: the triangle tests of the leaf children that a step hits are
// queued per warp in shared memory as (leaf slot, lane) and run by all 32
// lanes once kLeafFlush are queued (or when no lane can go on without their
// outcome).  Each test folds its hit into the owner's (t, id) key with one
// shared-memory atomicMin; the closest (t, id) over the tested triangles does
// not depend on the order of the tests, and the culling distance only lags.
// Tests where the traversal met them, whole warps waiting for their longest
// ray, and branches for push and pop left 12 of 32 lanes active; now 23 are.
// 1,048,576 rays on 262,144 triangles: 2.64 -> 1.92 ms (L1's data pipe is
// 86 % busy: load_child); 4.0 M rays on 4.2 M triangles 9.33 -> 5.64 ms;
// 77.5 M rays over 4,096 meshes 48.5 -> 31.6 ms.  Flush at 8 / 12 / 16 / 20 /
// 24 tests: 1.91 / 1.93 / 1.94 / 1.96 / 2.03 ms; 1 / 2 / 4 / 6 / 8 node steps
// between two looks at refill, flush and finished rays: 2.08 / 2.05 / 1.93 /
// 1.92 / 2.10 ms.  Once there are no more rays to take, a warp's time is that
// of its longest ray, and the looks are part of it: 6 / 10 / 16 / 24 steps from
// then on take 146 / 143 / 142 / 143 us for 170,001 rays on 5,001 triangles.
// Shared memory decides how much of it L1 keeps: 18 KB per CTA at 8 CTAs leaves
// 64 KB; 22 KB at 9 CTAs leaves next to none, and the 4.2 M triangles took 11.7
// ms.
constexpr int kLeafFlush = 12;
constexpr int kSteps = 6;  // node steps between two looks at what else is to be done
constexpr int kStepsLast = 24;  // the same, once there are no more rays to take
constexpr int kLeafQueue = 96;  // a step queues at most 64

template <bool BATCHED, bool V8, int REFILL>
__global__ void __launch_bounds__(kTraceThreads, kTraceCtas) k_trace_closest(const TraceArgs A) {
  __shared__ float2 s_stack[kStackShared][kTraceThreads];
  __shared__ RefineQueue s_rq[kTraceWarps];
  __shared__ uint32_t s_qslot[kTraceWarps][kLeafQueue];
  __shared__ uint8_t s_qlane[kTraceWarps][kLeafQueue];
  __shared__ unsigned long long s_best[kTraceWarps][32];
  __shared__ uint32_t s_bslot[kTraceWarps][32];
  // what only the triangle tests and the final store read
  __shared__ float s_rs[kTraceWarps][4][32];  // Sx, Sy, Sz, tmax of each lane's ray
  __shared__ int s_rk[kTraceWarps][32];       // kx | ky << 2 | kz << 4
  __shared__ unsigned long long s_rid[kTraceWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  RefineQueue &rq = s_rq[w];
  uint32_t *qslot = s_qslot[w];
  uint8_t *qlane = s_qlane[w];
  unsigned long long *sbest = s_best[w];
  bool active = false, drained = false, pending = false;
  RayPairs P;
  P.nxy = P.nzz = P.ixy = P.izz = 0;
  P.tmin = 0.0f;
  float bt = 0.0f;
  uint32_t base_leaf = 0, base_node = 0;
  int nq = 0, nrq = 0;  // queued tests, queued hits: the same on every lane
  Walk W;
  W.start();
  W.node = -1;
  float2 *const sh = &s_stack[0][threadIdx.x];
  float2 over[kStackDepth - kStackShared];

  // every queued test by all lanes (warp-uniform call)
  auto flush = [&]() {
    __syncwarp();
    for (int b = 0; b < nq; b += 32) {
      const int e = b + lane;
      const bool on = e < nq;
      const uint32_t slot = on ? qslot[e] : 0u;
      const int o = on ? qlane[e] : lane;
      float nx, ny, nz, unused;
      up2(__shfl_sync(FULL_MASK, P.nxy, o), nx, ny);
      up2(__shfl_sync(FULL_MASK, P.nzz, o), nz, unused);
      Ray Q;
      Q.ox = -nx;
      Q.oy = -ny;
      Q.oz = -nz;
      Q.tmin = __shfl_sync(FULL_MASK, P.tmin, o);
      Q.Sx = s_rs[w][0][o];
      Q.Sy = s_rs[w][1][o];
      Q.Sz = s_rs[w][2][o];
      Q.tmax = s_rs[w][3][o];
      const int k = s_rk[w][o];
      Q.kx = k & 3;
      Q.ky = (k >> 2) & 3;
      Q.kz = k >> 4;
      unsigned long long key = ~0ull;
      if (on) {
        const float4 a = __ldg(A.leaf + 3 * (size_t)slot), bb = __ldg(A.leaf + 3 * (size_t)slot + 1),
                     c = __ldg(A.leaf + 3 * (size_t)slot + 2);
        const float v0[3] = {a.x, a.y, a.z}, v1[3] = {bb.x, bb.y, bb.z}, v2[3] = {c.x, c.y, c.z};
        float t;
        if (isect_tri(Q, v0, v1, v2, t)) {
          key = ((unsigned long long)t_order(t) << 32) | __float_as_uint(a.w);
          atomicMin(&sbest[o], key);
        }
      }
      __syncwarp();
      if (key != ~0ull && sbest[o] == key) s_bslot[w][o] = slot;  // one winner per owner
      __syncwarp();
    }
    if (pending) {
      bt = t_from_order((uint32_t)(sbest[lane] >> 32));
      pending = false;
    }
    nq = 0;
  };
  // queue this lane's leaf (if it has one) 
  auto queue = [&](bool leaf, uint32_t slot) {
    const unsigned m = __ballot_sync(FULL_MASK, leaf);
    if (!m) return;
    if (leaf) {
      const int k = nq + __popc(m & lt);
      qslot[k] = slot;
      qlane[k] = (uint8_t)lane;
      pending = true;
    }
    nq += __popc(m);
  };

  while (true) {
    {
      uint64_t r;
      uint32_t n;
      Ray R;
      bool one = false;
      if (take_rays<BATCHED, REFILL>(A, active, drained, r, R, n, base_leaf, base_node)) {
        active = true;
        P = ray_pairs(R);
        bt = R.tmax;
        W.start();
        sbest[lane] = ((unsigned long long)t_order(R.tmax) << 32) | kMiss;
        s_rs[w][0][lane] = R.Sx;
        s_rs[w][1][lane] = R.Sy;
        s_rs[w][2][lane] = R.Sz;
        s_rs[w][3][lane] = R.tmax;
        s_rk[w][lane] = R.kx | (R.ky << 2) | (R.kz << 4);
        s_rid[w][lane] = r;
        if (n == 1) {
          one = single_leaf_box(A.leaf, base_leaf, R);
          W.node = -1;
        }
      }
      if (!__any_sync(FULL_MASK, active)) {
        if (drained) break;
        continue;
      }
      if (nq > kLeafQueue - 32) flush();
      queue(one, base_leaf);
    }
#pragma unroll 1
    for (int step = 0; step < (drained ? kStepsLast : kSteps); ++step) {
      const bool on = W.node >= 0;
      float t0 = __int_as_float(0x7fffffff), t1 = t0;
      int r0 = 0, r1 = 0;
      bool leaf0 = false, leaf1 = false;
      if (on && W.t <= bt) {
        const Bvh2Node *nd = A.bvh + base_node + W.node;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        t0 = child_entry(c0, P, bt);
        t1 = child_entry(c1, P, bt);
        r0 = c0.ref;
        r1 = c1.ref;
        leaf0 = r0 < 0 && t0 == t0;
        leaf1 = r1 < 0 && t1 == t1;
        if (r0 < 0) t0 = __int_as_float(0x7fffffff);
        if (r1 < 0) t1 = __int_as_float(0x7fffffff);
      }
      if (!walk_next<kTraceThreads, kStackShared, kStackDepth>(W, sh, over, on, t0, r0, t1, r1)) {
        atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
        W.node = -1;
      }
      if (__any_sync(FULL_MASK, leaf0 || leaf1)) {
        if (nq > kLeafQueue - 64) flush();
        queue(leaf0, base_leaf + (uint32_t)~r0);
        queue(leaf1, base_leaf + (uint32_t)~r1);
      }
    }
    const bool done = W.node < 0;
    const unsigned waiting = __ballot_sync(FULL_MASK, done && active && pending);
    const unsigned running = __ballot_sync(FULL_MASK, active && !done);
    if (nq >= kLeafFlush || (waiting && (!running || A.lanes - __popc(running) >= REFILL))) flush();
    const bool fin = active && done && !pending;
    if (__any_sync(FULL_MASK, fin)) {
      const bool hit = fin && (uint32_t)sbest[lane] != kMiss;
      finish_rays(A, rq, nrq, fin, hit, s_rid[w][lane], s_bslot[w][lane]);
      if (fin) active = false;
    }
  }
  refine_queued(A, rq, 0, nrq);
}

// The triangle tests of pool_walk (few rays) and what they need of a ray
// besides its origin, reciprocal direction, tmin and tmax.
struct PoolTriangles {
  const float4 *leaf;
  float4 *shear;  // per ray {Sx, Sy, Sz, kx | ky << 2 | kz << 4}
  uint32_t *slot;  // leaf slot of each ray's best hit
  __device__ __forceinline__ unsigned long long test(uint32_t s, int ray, const float4 &o, const float4 &i,
                                                     float &) const {
    const float4 q = shear[ray];
    Ray Q;
    Q.ox = -o.x;
    Q.oy = -o.y;
    Q.oz = -o.z;
    Q.tmin = o.w;
    Q.tmax = i.w;
    Q.Sx = q.x;
    Q.Sy = q.y;
    Q.Sz = q.z;
    const int k = __float_as_int(q.w);
    Q.kx = k & 3;
    Q.ky = (k >> 2) & 3;
    Q.kz = k >> 4;
    const float4 a = __ldg(leaf + 3 * (size_t)s), b = __ldg(leaf + 3 * (size_t)s + 1),
                 c = __ldg(leaf + 3 * (size_t)s + 2);
    const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
    float t;
    if (!isect_tri(Q, v0, v1, v2, t)) return ~0ull;
    return ((unsigned long long)t_order(t) << 32) | __float_as_uint(a.w);
  }
  __device__ __forceinline__ void won(int ray, uint32_t s, float) const { slot[ray] = s; }
};

template <bool BATCHED, bool V8>
__global__ void __launch_bounds__(kPoolThreads, kPoolCtas) k_trace_pool(const TraceArgs A) {
  __shared__ PoolShared s_pool[kPoolWarps];
  __shared__ float4 s_shear[kPoolWarps][kPoolRays];
  __shared__ uint32_t s_bslot[kPoolWarps][kPoolRays];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  PoolShared &S = s_pool[w];
  const PoolTriangles tris{A.leaf, s_shear[w], s_bslot[w]};
  while (true) {
    unsigned long long first = 0;
    if (lane == 0) first = atomicAdd(A.counter, (unsigned long long)A.lanes);
    first = __shfl_sync(FULL_MASK, first, 0);
    if (first >= A.nrays) break;
    const uint64_t r = first + lane;
    const bool mine = lane < A.lanes && r < A.nrays;
    bool one = false, root = false;
    uint32_t base_leaf = 0, base_node = 0;
    if (mine) {
      Ray R;
      ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
      uint32_t n = A.n;
      if (BATCHED) {
        const uint32_t m = mesh_of_ray(A.tm, r);
        base_leaf = __ldg(A.tm.tri_off + m);
        n = __ldg(A.tm.tri_off + m + 1) - base_leaf;
        base_node = base_leaf - m;
      }
      pool_ray(S, lane, R, base_leaf, base_node);
      s_shear[w][lane] = make_float4(R.Sx, R.Sy, R.Sz, __int_as_float(R.kx | (R.ky << 2) | (R.kz << 4)));
      root = n > 1;
      one = n == 1 && single_leaf_box(A.leaf, base_leaf, R);
    }
    if (!pool_walk<BATCHED, V8>(S, A.bvh, root, one, tris)) {
      if (lane == 0) atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
      break;
    }
    if (mine) {
      const unsigned long long key = S.best[lane];
      Hit h;
      h.prim = (uint32_t)key;
      h.t = __int_as_float(0x7f800000);
      if (h.prim != kMiss) {
        const uint32_t slot = s_bslot[w][lane];
        const float4 o = __ldg(A.rays + 2 * r), d = __ldg(A.rays + 2 * r + 1);
        Ray R;
        R.ox = o.x; R.oy = o.y; R.oz = o.z;
        R.dx = d.x; R.dy = d.y; R.dz = d.z;
        const float4 a = __ldg(A.leaf + 3 * (size_t)slot), b = __ldg(A.leaf + 3 * (size_t)slot + 1),
                     c = __ldg(A.leaf + 3 * (size_t)slot + 2);
        const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
        h.t = refine_t(R, v0, v1, v2);
      }
      A.hits[r] = h;
    }
    __syncwarp();
  }
}

}  // namespace gprtcu

using namespace gprtcu;

namespace {

gprtcuStatus trace_launch(const gprtcuLbvh *bvh, const uint32_t *tri_off, const uint32_t *ray_off, uint32_t meshes,
                          const float *rays, uint64_t nrays, gprtcuHit *hits, bool any, void *scratch,
                          size_t scratch_bytes, cudaStream_t stream) {
  if (!bvh || (!rays && nrays) || (!hits && nrays)) return GPRTCU_ERR_INVALID_ARG;
  if (meshes == 0 || (meshes > 1 && (!tri_off || !ray_off))) return GPRTCU_ERR_INVALID_ARG;
  if (nrays == 0) return GPRTCU_OK;
  if (bvh->numPrims == 0 || !bvh->leafTris || (bvh->numPrims > meshes && !bvh->bvh2)) return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)rays & 15) || ((uintptr_t)bvh->leafTris & 15) || ((uintptr_t)bvh->bvh2 & 15))
    return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  if (scratch_bytes < sizeof(ScratchHeader)) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  ScratchHeader *hdr = (ScratchHeader *)scratch;
  unsigned long long *counter = reinterpret_cast<unsigned long long *>(&hdr->ticket[0]);
  GPRTCU_TRY(cudaMemsetAsync(scratch, 0, sizeof(ScratchHeader), stream));
  const RayGrid g = ray_grid(nrays, kTraceCtas, kTraceWarps);
  TraceArgs a;
  a.bvh = (const Bvh2Node *)bvh->bvh2;
  a.leaf = (const float4 *)bvh->leafTris;
  a.n = bvh->numPrims;
  a.tm = TraceMeshes{tri_off, ray_off, meshes};
  a.rays = (const float4 *)rays;
  a.nrays = nrays;
  a.lanes = g.lanes;
  a.hits = (Hit *)hits;
  a.counter = counter;
  a.err = &hdr->status;
  const bool v8 = ((uintptr_t)bvh->bvh2 & 31) == 0;
  auto launch_any = [&](auto kernel) {
    cudaLaunchAttribute carveout;
    carveout.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    carveout.val.sharedMemCarveout = kAnyCarveout;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.ctas);
    cfg.blockDim = dim3(kTraceThreads);
    cfg.stream = stream;
    cfg.attrs = &carveout;
    cfg.numAttrs = g.ctas <= gprtcu_num_sms() * kAnyFewCtas ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, a);  // its error is taken up below
  };
  auto walk = [&](auto refill) {
    constexpr int F = decltype(refill)::value;
    auto launch = [&](auto kernel) { kernel<<<g.ctas, kTraceThreads, 0, stream>>>(a); };
    if (any) v8 ? launch_any(k_trace_any<false, true, F>) : launch_any(k_trace_any<false, false, F>);
    else v8 ? launch(k_trace_closest<false, true, F>) : launch(k_trace_closest<false, false, F>);
  };
  auto walk_batch = [&]() {
    auto launch = [&](auto kernel) { kernel<<<g.ctas, kTraceThreads, 0, stream>>>(a); };
    constexpr int F = kBatchRefill;
    if (any) v8 ? launch_any(k_trace_any<true, true, F>) : launch_any(k_trace_any<true, false, F>);
    else v8 ? launch(k_trace_closest<true, true, F>) : launch(k_trace_closest<true, false, F>);
  };
  // The pool (closest hit) while it is the faster form: up to 9/6 chunks per
  // warp, 85,248 rays on 148 SMs, and for meshes below 2,048 triangles, whose
  // walks are short, 6/6.  Plain walk / pool / lane per ray, us: 735 triangles and
  // 60,001 rays 41.6 / 41.5 / 39.0, 80,001 45.6 / 47.3 / 43.3; 2,657 triangles
  // 60,001 64.8 / 61.8 / 65.2, 80,001 72.1 / 70.4 / 72.2, 94,001 73.2 / 76.6 /
  // 72.2; 100,001 triangles 80,001 275 / 221 / 236, 113,001 312 / 265 / 262.
  const int pool_sixths = bvh->numPrims / meshes < 2048 ? 6 : 9;
  if (const RayGrid few = pool_grid(nrays, pool_sixths); !any && few.lanes) {
    a.lanes = few.lanes;
    auto launch = [&](auto kernel) { kernel<<<few.ctas, kPoolThreads, 0, stream>>>(a); };
    if (meshes > 1) v8 ? launch(k_trace_pool<true, true>) : launch(k_trace_pool<true, false>);
    else v8 ? launch(k_trace_pool<false, true>) : launch(k_trace_pool<false, false>);
  } else if (meshes > 1) {
    walk_batch();
  } else {
    switch (trace_refill(bvh->numPrims)) {
      case 32: walk(std::integral_constant<int, 32>()); break;
      case 24: walk(std::integral_constant<int, 24>()); break;
      default: walk(std::integral_constant<int, kTraceRefill>()); break;
    }
  }
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

}  // namespace

extern "C" GPRTCU_API size_t gprtcuTraceScratchSize(void) { return sizeof(ScratchHeader); }

extern "C" GPRTCU_API gprtcuStatus gprtcuTraceClosest(const gprtcuLbvh *bvh, const float *rays, uint64_t numRays,
                                                      gprtcuHit *hits, void *scratch, size_t scratchBytes,
                                                      gprtcuStream stream) {
  return trace_launch(bvh, nullptr, nullptr, 1, rays, numRays, hits, false, scratch, scratchBytes, (cudaStream_t)stream);
}

extern "C" GPRTCU_API gprtcuStatus gprtcuTraceAny(const gprtcuLbvh *bvh, const float *rays, uint64_t numRays,
                                                  gprtcuHit *hits, void *scratch, size_t scratchBytes,
                                                  gprtcuStream stream) {
  return trace_launch(bvh, nullptr, nullptr, 1, rays, numRays, hits, true, scratch, scratchBytes, (cudaStream_t)stream);
}

extern "C" GPRTCU_API gprtcuStatus gprtcuBatchTrace(const gprtcuLbvh *bvh, const uint32_t *triOffsets,
                                                    const uint32_t *rayOffsets, uint32_t numMeshes, const float *rays,
                                                    uint64_t numRays, int anyHit, gprtcuHit *hits, void *scratch,
                                                    size_t scratchBytes, gprtcuStream stream) {
  return trace_launch(bvh, triOffsets, rayOffsets, numMeshes, rays, numRays, hits, anyHit != 0, scratch, scratchBytes,
                      (cudaStream_t)stream);
}
