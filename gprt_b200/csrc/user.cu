// user.cu -- spheres and linearly swept spheres (LSS) as software-BVH
// primitives: their bounds, and closest-hit / any-hit traversal of an LBVH
// built over those bounds (gprtcuLbvhBuildBoxes) with the reference's
// ray/LSS intersection at the leaves.
//
// The reference traces these primitives on ray-tracing hardware: an AABB
// acceleration structure over the boxes of its SphereBounds / LSSBounds
// compute programs (gprt/gprt_fallbacks.slang:215-235,263-283), with
// SphereIntersection / LSSIntersection as intersection programs (:146-166,
// 245-261), both calling intersectRayLSS (:45-144).  Here the same arithmetic
// runs in CUDA: every float operation is an explicit round-to-nearest
// intrinsic in the reference's evaluation order (dot(a, b) = (a.x*b.x +
// a.y*b.y) + a.z*b.z, rcp(x) = 1/x), so bounds, t and u are bit-identical to
// the reference's code compiled for the host.
//
// Closest hit: the smallest t in the ray's (tmin, tmax), ties to the lowest
// primitive id (the reference's hardware leaves tie order unspecified); any
// hit: the first hit found.
#include "bvh2.cuh"
#include "common.cuh"
#include "lbvh.cuh"
#include "rtmath.cuh"

namespace gprtcu {

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 add3(F3 a, F3 b) { return f3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ F3 sub3(F3 a, F3 b) { return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ float dot3(F3 a, F3 b) {
  return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}

// intersectRayLSS (gprt/gprt_fallbacks.slang:45-144).
__device__ bool lss_intersect(F3 ro, F3 d, F3 p0, F3 p1, float r0, float r1, bool cap0, bool cap1, float tmin,
                              float tmax, bool exit_test, float &t_out, float &u_out) {
  t_out = 0.0f;
  u_out = 0.0f;
  const F3 mid = f3(__fmul_rn(0.5f, __fadd_rn(p0.x, p1.x)), __fmul_rn(0.5f, __fadd_rn(p0.y, p1.y)),
                    __fmul_rn(0.5f, __fadd_rn(p0.z, p1.z)));
  const float rmid = __fmul_rn(0.5f, __fadd_rn(r0, r1));
  const float dd = dot3(d, d);
  const float inv_dd = __fdiv_rn(1.0f, dd);
  const float align = __fmul_rn(dot3(d, sub3(mid, ro)), inv_dd);
  ro = f3(__fadd_rn(ro.x, __fmul_rn(align, d.x)), __fadd_rn(ro.y, __fmul_rn(align, d.y)),
          __fadd_rn(ro.z, __fmul_rn(align, d.z)));
  const F3 off = sub3(ro, mid);
  const F3 axis = sub3(p1, p0);
  const float rdel = __fsub_rn(r1, r0);
  const float a = dd;
  const float b = dot3(axis, d);
  const float c = __fsub_rn(dot3(axis, axis), __fmul_rn(rdel, rdel));
  const float dq = dot3(d, off);
  const float e = __fadd_rn(dot3(axis, off), __fmul_rn(rmid, rdel));
  const float f = __fsub_rn(dot3(off, off), __fmul_rn(rmid, rmid));
  const float At = __fsub_rn(__fmul_rn(b, b), __fmul_rn(a, c));
  const float Bt = __fsub_rn(__fmul_rn(b, e), __fmul_rn(c, dq));
  const float Ct = __fsub_rn(__fmul_rn(e, e), __fmul_rn(c, f));
  const float disc = __fsub_rn(__fmul_rn(Bt, Bt), __fmul_rn(At, Ct));
  const bool is_sphere = axis.x == 0.0f && axis.y == 0.0f && axis.z == 0.0f && rdel == 0.0f;
  const bool use_start_sphere = !cap1;
  const bool shell_degenerate = (c <= 0.0f) && (rdel != 0.0f);
  const bool invalid = (r0 <= 0.0f && r1 <= 0.0f) || isnan(r0) || isnan(r1) || isnan(p0.x) || isnan(p1.x) ||
                       isinf(r0) || isinf(p0.x);
  if ((!is_sphere && !shell_degenerate && disc < 0.0f) || invalid) return false;
  const float sq = __fsqrt_rn(disc);
  const float inv_at = __fdiv_rn(1.0f, At);
  const float t0 = __fmul_rn(__fadd_rn(-Bt, exit_test ? -sq : sq), inv_at);
  const float inv_c = __fdiv_rn(1.0f, c);
  const float u0 = __fmul_rn(__fadd_rn(__fmul_rn(b, t0), e), inv_c);
  if (fabsf(u0) <= 0.5f && (__fmul_rn(u0, rdel) >= -rmid) && !is_sphere && !shell_degenerate) {
    const float ht = __fadd_rn(t0, align), hu = __fadd_rn(u0, 0.5f);
    if (ht <= tmin || ht >= tmax) return false;
    t_out = ht;
    u_out = hu;
    return true;
  }
  const bool start_cap = is_sphere ? use_start_sphere : (u0 < 0.0f);
  if ((start_cap && !cap0) || (!start_cap && !cap1)) return false;
  const float Bs = __fadd_rn(-dq, __fmul_rn(start_cap ? -b : b, 0.5f));
  const float BsBs = __fmul_rn(Bs, Bs);
  const float Cs = __fsub_rn(__fadd_rn(f, __fmul_rn(0.25f, c)), start_cap ? -e : e);
  const float AsCs = __fmul_rn(a, Cs);
  if (BsBs < AsCs) return false;
  const float sqc = __fsqrt_rn(__fsub_rn(BsBs, AsCs));
  const float cap_t = __fmul_rn(__fsub_rn(Bs, exit_test ? -sqc : sqc), inv_dd);
  t_out = __fadd_rn(cap_t, align);
  u_out = start_cap ? 0.0f : 1.0f;
  if (t_out <= tmin || t_out >= tmax) return false;
  return true;
}

// One end of computeLssAabb: the box of end v (radius r, cap on/off) given
// the other end's data.
__device__ __forceinline__ void lss_end_box(F3 v, float r, bool cap, F3 v0, F3 v1, float r0, float r1, F3 cme, F3 cpe,
                                            F3 &lo, F3 &hi) {
  lo = v;
  hi = v;
  if (r < 0.0f) {
    const float s = __fmul_rn(r, __fdiv_rn(1.0f, __fsub_rn(r1, r0)));
    lo = f3(__fadd_rn(lo.x, __fmul_rn(s, __fsub_rn(v0.x, v1.x))), __fadd_rn(lo.y, __fmul_rn(s, __fsub_rn(v0.y, v1.y))),
            __fadd_rn(lo.z, __fmul_rn(s, __fsub_rn(v0.z, v1.z))));
    hi = lo;
  } else if (cap) {
    lo = f3(__fadd_rn(lo.x, -r), __fadd_rn(lo.y, -r), __fadd_rn(lo.z, -r));
    hi = f3(__fadd_rn(hi.x, r), __fadd_rn(hi.y, r), __fadd_rn(hi.z, r));
  } else {
    lo = f3(__fadd_rn(lo.x, __fmul_rn(r, cme.x)), __fadd_rn(lo.y, __fmul_rn(r, cme.y)), __fadd_rn(lo.z, __fmul_rn(r, cme.z)));
    hi = f3(__fadd_rn(hi.x, __fmul_rn(r, cpe.x)), __fadd_rn(hi.y, __fmul_rn(r, cpe.y)), __fadd_rn(hi.z, __fmul_rn(r, cpe.z)));
  }
}

// computeLssAabb (gprt/gprt_fallbacks.slang:168-213).
__device__ void lss_aabb(F3 v0, float r0, bool cap0, F3 v1, float r1, bool cap1, float *out) {
  F3 cme = f3(0.f, 0.f, 0.f), cpe = f3(0.f, 0.f, 0.f);
  if (!cap0 || !cap1) {
    const float rd = __fsub_rn(r1, r0);
    const F3 n = sub3(v0, v1);
    const F3 nsq = f3(__fmul_rn(n.x, n.x), __fmul_rn(n.y, n.y), __fmul_rn(n.z, n.z));
    const float l2 = __fadd_rn(__fadd_rn(nsq.x, nsq.y), nsq.z);
    const float l2inv = __fdiv_rn(1.0f, l2);
    const F3 X = f3(__fsub_rn(1.f, __fmul_rn(nsq.x, l2inv)), __fsub_rn(1.f, __fmul_rn(nsq.y, l2inv)),
                    __fsub_rn(1.f, __fmul_rn(nsq.z, l2inv)));
    const float Y = __fsub_rn(1.f, __fmul_rn(__fmul_rn(rd, rd), l2inv));
    const F3 e = f3(__fsqrt_rn(fabsf(__fmul_rn(X.x, Y))), __fsqrt_rn(fabsf(__fmul_rn(X.y, Y))),
                    __fsqrt_rn(fabsf(__fmul_rn(X.z, Y))));
    const F3 c = f3(__fmul_rn(__fmul_rn(rd, n.x), l2inv), __fmul_rn(__fmul_rn(rd, n.y), l2inv),
                    __fmul_rn(__fmul_rn(rd, n.z), l2inv));
    cme = sub3(c, e);
    cpe = add3(c, e);
  }
  F3 lo0, hi0, lo1, hi1;
  lss_end_box(v0, r0, cap0, v0, v1, r0, r1, cme, cpe, lo0, hi0);
  lss_end_box(v1, r1, cap1, v0, v1, r0, r1, cme, cpe, lo1, hi1);
  out[0] = fminf(lo0.x, lo1.x);
  out[1] = fminf(lo0.y, lo1.y);
  out[2] = fminf(lo0.z, lo1.z);
  out[3] = fmaxf(hi0.x, hi1.x);
  out[4] = fmaxf(hi0.y, hi1.y);
  out[5] = fmaxf(hi0.z, hi1.z);
}

// SphereBounds (gprt/gprt_fallbacks.slang:263-283).
__global__ void k_sphere_bounds(const float4 *spheres, uint32_t n, float *aabbs) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 s = spheres[i];
    const float r = fmaxf(s.w, 0.0f);
    const float c[3] = {s.x, s.y, s.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      aabbs[6 * (size_t)i + k] = fminf(3.402823466e38f, __fsub_rn(c[k], r));
      aabbs[6 * (size_t)i + 3 + k] = fmaxf(-3.402823466e38f, __fadd_rn(c[k], r));
    }
  }
}

// LSSBounds (gprt/gprt_fallbacks.slang:215-235).
__global__ void k_lss_bounds(const float4 *verts, const uint2 *idx, uint32_t n, int cap0, int cap1, float *aabbs) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint2 e = idx[i];
    const float4 a = verts[e.x], b = verts[e.y];
    lss_aabb(f3(a.x, a.y, a.z), a.w, cap0 != 0, f3(b.x, b.y, b.z), b.w, cap1 != 0, aabbs + 6 * (size_t)i);
  }
}

// Primitive access: a sphere is the LSS with both ends equal and both caps on
// (SphereIntersection, gprt/gprt_fallbacks.slang:245-261).
struct SpherePrims {
  const float4 *spheres;
  // only o, d, tmin and tmax of the ray are read
  __device__ __forceinline__ bool hit(const Ray &R, uint32_t id, bool exit_test, float &t, float &u) const {
    const float4 s = __ldg(spheres + id);
    const F3 c = f3(s.x, s.y, s.z);
    return lss_intersect(f3(R.ox, R.oy, R.oz), f3(R.dx, R.dy, R.dz), c, c, s.w, s.w, true, true, R.tmin, R.tmax,
                         exit_test, t, u);
  }
};
struct LssPrims {
  const float4 *verts;
  const uint2 *idx;
  bool cap0, cap1;
  __device__ __forceinline__ bool hit(const Ray &R, uint32_t id, bool exit_test, float &t, float &u) const {
    const uint2 e = __ldg(idx + id);
    const float4 a = __ldg(verts + e.x), b = __ldg(verts + e.y);
    return lss_intersect(f3(R.ox, R.oy, R.oz), f3(R.dx, R.dy, R.dz), f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), a.w, b.w,
                         cap0, cap1, R.tmin, R.tmax, exit_test, t, u);
  }
};

template <typename PRIMS> struct UserArgs {
  const Bvh2Node *bvh;
  const uint32_t *ids;
  uint32_t n;
  const float *root_box;
  PRIMS prims;
  bool exit_test;
  const float4 *rays;
  uint64_t nrays;
  int lanes;  // rays a warp holds at a time
  Hit *hits;
  float *hit_u;
  unsigned long long *counter;
  uint32_t *err;
};

constexpr int kUserThreads = 128;
constexpr int kUserWarps = kUserThreads / 32;
constexpr int kUserShared = 12;  // stack entries in shared memory
constexpr int kUserDepth = 64;
constexpr int kUserRefill = 8;
constexpr int kUserSteps = 14;
constexpr int kUserFlush = 12;
constexpr int kUserQueue = 96;  // a step queues at most 64

// A ray whose closest hit so far is no number (an infinite or NaN coordinate,
// or no direction, can give a primitive test a distance that is NaN): such a
// hit is the ray's last, and only counts when it is the ray's first, so the
// order of the tests decides.  The traversals mark it with a key below every
// distance's (odd_key; it also ends the walk, since nothing compares with its
// NaN), and the ray is walked again here, one test after the other, nearer
// child first.  (Folded in as an ordinary key such a hit was lost and the walk
// went on over every primitive: 1,048,577 rays on 1,048,576 swept spheres with
// one component in twenty infinite, NaN, zero or huge took 866 ms instead of
// 2.2 ms.)
constexpr unsigned long long kOddKey = 0;
__device__ __forceinline__ bool odd_key(unsigned long long key) { return (uint32_t)(key >> 32) < t_order(-INFINITY); }
__device__ __forceinline__ unsigned long long hit_key(float t, uint32_t id) {
  return t == t ? ((unsigned long long)t_order(t) << 32) | id : kOddKey;
}
template <typename PRIMS> __device__ __forceinline__ void user_odd(const UserArgs<PRIMS> &A, uint64_t r) {
  Ray R;
  ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
  uint32_t best = kMiss;
  float bt = R.tmax, bu = 0.0f;
  auto leaf = [&](uint32_t slot) {
    const uint32_t id = __ldg(A.ids + slot);
    float t, u;
    if (A.prims.hit(R, id, A.exit_test, t, u) && (best == kMiss || t < bt || (t == bt && id < best))) {
      best = id;
      bt = t;
      bu = u;
    }
  };
  auto entry = [&](const Bvh2Child &c, float &tn) {
    return ray_box(R, c.box[0], c.box[1], c.box[4], c.box[2], c.box[3], c.box[5], bt, tn) && tn <= bt;
  };
  int stack[kUserDepth];
  int sp = 0, node = 0;
  float tn0, tn1;
  if (A.n == 1) {
    if (ray_box(R, A.root_box[0], A.root_box[1], A.root_box[2], A.root_box[3], A.root_box[4], A.root_box[5], bt, tn0))
      leaf(0);
  }
  while (A.n > 1) {
    const Bvh2Node &nd = A.bvh[node];
    const int r0 = nd.c[0].ref, r1 = nd.c[1].ref;
    bool h0 = entry(nd.c[0], tn0), h1 = entry(nd.c[1], tn1);
    if (h0 && r0 < 0) leaf((uint32_t)~r0);
    h1 = h1 && tn1 <= bt;
    if (h1 && r1 < 0) leaf((uint32_t)~r1);
    h0 = h0 && r0 >= 0;
    h1 = h1 && r1 >= 0 && tn1 <= bt;
    if (h0 && h1) {
      const bool first0 = tn0 <= tn1;
      if (sp == kUserDepth) {
        atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
        break;
      }
      stack[sp++] = first0 ? r1 : r0;
      node = first0 ? r0 : r1;
    } else if (h0 || h1) {
      node = h0 ? r0 : r1;
    } else if (sp > 0) {
      node = stack[--sp];
    } else {
      break;
    }
  }
  Hit h;
  h.prim = best;
  h.t = best == kMiss ? __int_as_float(0x7f800000) : bt;
  A.hits[r] = h;
  if (A.hit_u) A.hit_u[r] = best == kMiss ? 0.0f : bu;
}
// Writes the hit of ray r from its closest (t, id) and that hit's u.  An odd
// ray is put on the lane's list instead (its hit holds the list's next ray),
// which the lane goes through at its end: called where hits are written,
// user_odd made the traversals spill.
constexpr unsigned long long kOddEnd = ~0ull;
__device__ __forceinline__ float2 odd_link(unsigned long long r) {
  return make_float2(__uint_as_float((uint32_t)r), __uint_as_float((uint32_t)(r >> 32)));
}
template <typename PRIMS>
__device__ __forceinline__ void user_hit(const UserArgs<PRIMS> &A, uint64_t r, unsigned long long key, float u,
                                         float2 &odd) {
  Hit h;
  if (odd_key(key)) {
    h.prim = __float_as_uint(odd.x);
    h.t = odd.y;
    A.hits[r] = h;
    odd = odd_link(r);
    return;
  }
  const bool hit = (uint32_t)key != kMiss;
  h.prim = (uint32_t)key;
  h.t = hit ? t_from_order((uint32_t)(key >> 32)) : __int_as_float(0x7f800000);
  A.hits[r] = h;
  if (A.hit_u) A.hit_u[r] = hit ? u : 0.0f;
}
template <typename PRIMS>
__device__ __forceinline__ void user_odds(const UserArgs<PRIMS> &A, float2 odd) {
  while (true) {
    const uint64_t r = ((unsigned long long)__float_as_uint(odd.y) << 32) | __float_as_uint(odd.x);
    if (r == kOddEnd) break;
    const Hit h = A.hits[r];
    odd = make_float2(__uint_as_float(h.prim), h.t);
    user_odd(A, r);
  }
}

// Binary LBVH traversal (the layout of gprtcuLbvh.bvh2) with the primitive
// test at the leaves: leaf slot s holds primitive ids[s].  One lane per ray,
// refilled as rays finish.  Closest hit queues the tests of the leaf children
// it meets per warp as (slot, lane) and runs them with all lanes, each folding
// its hit into the owner's (t, id) key.  (A test is 150 to 200 instructions; run
// where the walk met them, with whole warps waiting for their longest ray,
// they left 8.4 of 32 lanes active.  1,048,577 rays on 1,048,576 swept
// spheres: 2.51 -> 1.45 ms; what bounds it now is load latency and L1's data
// pipe.  Flush at 8 / 12 / 24 / 32 tests: 1.56 / 1.56 / 1.60 / 1.66 ms, and from
// there 6 / 8 / 10 node steps between two looks at flush and refill with 8 / 8 /
// 12 stack entries in shared memory: 1.56 / 1.52 / 1.47 ms.)  With no more rays
// to take, a flush comes as soon as the lanes still walking have a test each:
// the culling distance lags less, which is worth more than full lanes then
// (130,001 rays on 1,000,001 spheres 549 -> 481 us; 500 in the plain walk).  7 /
// 8 CTAs per SM (72 / 64 registers, the latter spilling some 30 bytes): 130,001
// and 1,048,577 rays on a million spheres 481 / 507 us and 1.38 / 1.43 ms, on a
// million swept spheres 461 / 478 us and 1.48 / 1.45 ms, 4.2 M rays on 4.2 M
// swept spheres 4.82 / 4.55 ms: spheres run 7, swept spheres, which wait more on
// memory, 8.  6 CTAs: 1.43 ms on the million spheres.  10 / 14 node steps between
// two looks 1.47 / 1.45 ms on the million swept spheres.
template <typename PRIMS> constexpr int kUserCtas = 7;
template <> constexpr int kUserCtas<LssPrims> = 8;
template <typename PRIMS, bool V8>
__global__ void __launch_bounds__(kUserThreads, kUserCtas<PRIMS>) k_user_closest(const UserArgs<PRIMS> A) {
  __shared__ float2 s_stack[kUserShared][kUserThreads];
  __shared__ uint32_t s_qslot[kUserWarps][kUserQueue];
  __shared__ uint8_t s_qlane[kUserWarps][kUserQueue];
  __shared__ unsigned long long s_best[kUserThreads];  // closest (t, id)
  __shared__ float s_u[kUserThreads];                  // u of that hit
  __shared__ float s_dir[4][kUserThreads];             // direction, tmax
  __shared__ unsigned long long s_rid[kUserThreads];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, wbase = tid & ~31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t *qslot = s_qslot[w];
  uint8_t *qlane = s_qlane[w];
  const float kNone = __int_as_float(0x7fffffff);
  bool active = false, drained = false, pending = false;
  RayPairs P;
  P.nxy = P.nzz = P.ixy = P.izz = 0;
  P.tmin = 0.0f;
  float bt = 0.0f;
  int nq = 0;  // queued tests, the same on every lane
  Walk W;
  W.start();
  W.node = kWalkEnd;
  float2 *const sh = &s_stack[0][tid];
  float2 over[kUserDepth - kUserShared + 1];
  float2 &odd = over[kUserDepth - kUserShared];  // the lane's list of odd rays
  odd = odd_link(kOddEnd);

  // the primitive of a leaf slot against lane o's ray (its origin and tmin
  // given); true when it is hit, the key folded into that lane's best
  auto test = [&](uint32_t slot, int o, float ox, float oy, float oz, float tmin, float &u) -> unsigned long long {
    Ray Q;
    Q.ox = ox;
    Q.oy = oy;
    Q.oz = oz;
    Q.tmin = tmin;
    Q.dx = s_dir[0][wbase + o];
    Q.dy = s_dir[1][wbase + o];
    Q.dz = s_dir[2][wbase + o];
    Q.tmax = s_dir[3][wbase + o];
    const uint32_t id = __ldg(A.ids + slot);
    float t;
    if (!A.prims.hit(Q, id, A.exit_test, t, u)) return ~0ull;
    return hit_key(t, id);
  };
  // every queued test by all lanes (warp-uniform call)
  auto flush = [&]() {
    __syncwarp();
    for (int b = 0; b < nq; b += 32) {
      const int e = b + lane;
      const bool on = e < nq;
      const uint32_t slot = on ? qslot[e] : 0u;
      const int o = on ? qlane[e] : lane;
      float nx, ny, nz, unused, u;
      up2(__shfl_sync(FULL_MASK, P.nxy, o), nx, ny);
      up2(__shfl_sync(FULL_MASK, P.nzz, o), nz, unused);
      const float tmin = __shfl_sync(FULL_MASK, P.tmin, o);
      unsigned long long key = ~0ull;
      if (on) key = test(slot, o, -nx, -ny, -nz, tmin, u);
      if (key != ~0ull) atomicMin(&s_best[wbase + o], key);
      __syncwarp();
      if (key != ~0ull && s_best[wbase + o] == key) s_u[wbase + o] = u;  // one winner per owner
      __syncwarp();
    }
    if (pending) {
      bt = t_from_order((uint32_t)(s_best[tid] >> 32));
      pending = false;
    }
    nq = 0;
  };
  auto queue = [&](bool leaf, uint32_t slot) {
    const unsigned m = __ballot_sync(FULL_MASK, leaf);
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
      bool one = false;
      if (warp_take(active, drained, A.lanes, kUserRefill, A.nrays, A.counter, r)) {
        Ray R;
        ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
        active = true;
        P = ray_pairs(R);
        bt = R.tmax;
        W.start();
        s_best[tid] = ((unsigned long long)t_order(R.tmax) << 32) | kMiss;
        s_dir[0][tid] = R.dx;
        s_dir[1][tid] = R.dy;
        s_dir[2][tid] = R.dz;
        s_dir[3][tid] = R.tmax;
        s_rid[tid] = r;
        if (A.n == 1) {
          float tn;
          one = ray_box(R, A.root_box[0], A.root_box[1], A.root_box[2], A.root_box[3], A.root_box[4], A.root_box[5],
                        bt, tn);
          W.node = kWalkEnd;
        }
      }
      if (!__any_sync(FULL_MASK, active)) {
        if (drained) break;
        continue;
      }
      if (nq > kUserQueue - 32) flush();
      queue(one, 0u);
    }
#pragma unroll 1
    for (int step = 0; step < kUserSteps; ++step) {
      const bool on = W.node >= 0;
      float t0 = kNone, t1 = kNone;
      int r0 = 0, r1 = 0;
      bool leaf0 = false, leaf1 = false;
      if (on && W.t <= bt) {
        const Bvh2Node *nd = A.bvh + W.node;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        t0 = child_entry(c0, P, bt);
        t1 = child_entry(c1, P, bt);
        r0 = c0.ref;
        r1 = c1.ref;
        leaf0 = r0 < 0 && t0 == t0;
        leaf1 = r1 < 0 && t1 == t1;
        if (leaf0) t0 = kNone;
        if (leaf1) t1 = kNone;
      }
      if (!walk_next<kUserThreads, kUserShared, kUserDepth>(W, sh, over, on, t0, r0, t1, r1)) {
        atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
        W.node = kWalkEnd;
      }
      if (__any_sync(FULL_MASK, leaf0 || leaf1)) {
        if (nq > kUserQueue - 64) flush();
        queue(leaf0, (uint32_t)~r0);
        queue(leaf1, (uint32_t)~r1);
      }
    }
    const bool done = W.node == kWalkEnd;
    const unsigned waiting = __ballot_sync(FULL_MASK, done && active && pending);
    const unsigned running = __ballot_sync(FULL_MASK, active && !done);
    if (nq >= kUserFlush || (drained && nq >= __popc(running)) ||
        (waiting && (!running || A.lanes - __popc(running) >= kUserRefill)))
      flush();
    if (active && done && !pending) {
      user_hit(A, s_rid[tid], s_best[tid], s_u[tid], odd);
      active = false;
    }
  }
  user_odds(A, odd);
}

// Any hit (ANY): the primitives of the leaf children that a step meets are tested
// at once, child 0 first, and the first step with a hit ends the ray, as the
// any-hit walk over triangles does.  Ray and hit in registers and a stack of
// nodes alone (the closest-hit kernel with its tests at once kept them in
// shared memory, 17 KB a CTA): 30,001 / 1,000,001 rays on 1,000,001 swept
// spheres 344 / 1,697 -> 317 / 1,504 us, 150,001 rays on 10,001 spheres 149 ->
// 122 us.  Steps between two votes 12 / 12 and 48 once there are no more rays to
// take: 20,001 rays on 1,001 spheres 29 / 33 us.  Closest hit in the same form
// (few primitives: trace_user) culls by the best distance when it visits a
// node, not when it takes it off the stack, and keeps to the order of
// user_odd, so a hit at a distance that is no number needs no second walk.
constexpr int kUserAnyCtas = 8;
constexpr int kUserAnyShared = 8;  // stack entries (nodes alone) in shared memory
constexpr int kUserAnySteps = 12;
template <typename PRIMS, bool ANY, bool V8>
__global__ void __launch_bounds__(kUserThreads, kUserAnyCtas) k_user_lane(const UserArgs<PRIMS> A) {
  __shared__ int s_stack[kUserAnyShared][kUserThreads];
  bool active = false, drained = false;
  uint64_t r = 0;
  RayPairs P;
  P.nxy = P.nzz = P.ixy = P.izz = 0;
  P.tmin = 0.0f;
  float dx = 0.0f, dy = 0.0f, dz = 0.0f, tmax = 0.0f;
  uint32_t best = kMiss;
  float bt = 0.0f, bu = 0.0f;
  int node = -1, top = -1, sp = 0;  // the walk: its node, the stack's top entry and the entries below it
  int *const sh = &s_stack[0][threadIdx.x];
  int over[kUserDepth - kUserAnyShared];
  auto test = [&](uint32_t slot) {
    Ray Q;
    float nx, ny, nz, unused;
    up2(P.nxy, nx, ny);
    up2(P.nzz, nz, unused);
    Q.ox = -nx;
    Q.oy = -ny;
    Q.oz = -nz;
    Q.tmin = P.tmin;
    Q.dx = dx;
    Q.dy = dy;
    Q.dz = dz;
    Q.tmax = tmax;
    const uint32_t id = __ldg(A.ids + slot);
    float t, u;
    if (A.prims.hit(Q, id, A.exit_test, t, u) && (best == kMiss || t < bt || (t == bt && id < best))) {
      best = id;
      bt = t;
      bu = u;
    }
  };
  while (true) {
    if (warp_take(active, drained, A.lanes, kUserRefill, A.nrays, A.counter, r)) {
      Ray R;
      ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
      active = true;
      P = ray_pairs(R);
      dx = R.dx;
      dy = R.dy;
      dz = R.dz;
      bt = tmax = R.tmax;
      best = kMiss;
      node = bt == bt ? 0 : -1;  // no box lies in a range that ends in NaN
      top = -1;
      sp = 0;
      if (A.n == 1) {
        float tn;
        if (ray_box(R, A.root_box[0], A.root_box[1], A.root_box[2], A.root_box[3], A.root_box[4], A.root_box[5], bt,
                    tn))
          test(0);
        node = -1;
      }
    }
    if (!__any_sync(FULL_MASK, active)) {
      if (drained) break;
      continue;
    }
#pragma unroll 1
    for (int step = 0; step < kUserAnySteps; ++step) {
      if (node >= 0) {
        const Bvh2Node *nd = A.bvh + node;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        float t0, t1;
        const bool h0 = child_hit(c0, P, bt, t0), h1 = child_hit(c1, P, bt, t1);
        if (h0 && c0.ref < 0) test((uint32_t)~c0.ref);
        if (h1 && c1.ref < 0 && t1 <= bt) test((uint32_t)~c1.ref);
        const bool in0 = h0 && c0.ref >= 0, in1 = h1 && c1.ref >= 0 && (ANY || t1 <= bt);
        const bool first = in0 && !(in1 && t1 < t0);  // the nearer child, child 0 on ties
        if (ANY ? best != kMiss : bt != bt) {  // a hit at a distance that is no number is a ray's last
          node = -1;
        } else if (in0 || in1) {
          if (in0 && in1) {
            if (sp < kUserAnyShared) sh[sp * kUserThreads] = top;
            else if (sp < kUserDepth) over[sp - kUserAnyShared] = top;
            ++sp;
            top = first ? c1.ref : c0.ref;
          }
          node = first ? c0.ref : c1.ref;
          if (sp > kUserDepth) {
            atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
            node = -1;
          }
        } else {
          node = top;
          --sp;
          top = sp < 0 ? -1 : (sp < kUserAnyShared ? sh[sp * kUserThreads] : over[sp - kUserAnyShared]);
        }
      }
    }
    if (active && node < 0) {
      Hit h;
      h.prim = best;
      h.t = best == kMiss ? __int_as_float(0x7f800000) : bt;
      A.hits[r] = h;
      if (A.hit_u) A.hit_u[r] = best == kMiss ? 0.0f : bu;
      active = false;
    }
  }
}

// The primitive tests of pool_walk (few rays): the ray's direction, and u of
// its best hit, per ray.
template <typename PRIMS> struct PoolPrims {
  const UserArgs<PRIMS> &A;
  float4 *dir;
  float *u;
  __device__ __forceinline__ unsigned long long test(uint32_t s, int ray, const float4 &o, const float4 &i,
                                                     float &hu) const {
    const float4 d = dir[ray];
    Ray Q;
    Q.ox = -o.x;
    Q.oy = -o.y;
    Q.oz = -o.z;
    Q.tmin = o.w;
    Q.dx = d.x;
    Q.dy = d.y;
    Q.dz = d.z;
    Q.tmax = i.w;
    const uint32_t id = __ldg(A.ids + s);
    float t;
    if (!A.prims.hit(Q, id, A.exit_test, t, hu)) return ~0ull;
    return hit_key(t, id);
  }
  __device__ __forceinline__ void won(int ray, uint32_t, float hu) const { u[ray] = hu; }
};

template <typename PRIMS, bool V8>
__global__ void __launch_bounds__(kPoolThreads, kPoolCtas) k_user_pool(const UserArgs<PRIMS> A) {
  __shared__ PoolShared s_pool[kPoolWarps];
  __shared__ float4 s_dir[kPoolWarps][kPoolRays];
  __shared__ float s_u[kPoolWarps][kPoolRays];
  __shared__ float2 s_odd[kPoolWarps][kPoolRays];  // lists of odd rays
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  PoolShared &S = s_pool[w];
  const PoolPrims<PRIMS> prims{A, s_dir[w], s_u[w]};
  if (lane < kPoolRays) s_odd[w][lane] = odd_link(kOddEnd);
  // The shared visits meet the tests in another order than user_odd, and can
  // pass by a primitive that would give a distance that is no number: rays
  // for which one could, go there at once.  With m the larger of the distances
  // from zero of the ray's origin and the scene's farthest corner, all that
  // the last test of lss_intersect forms is below 100 m^2 |d|^2, 100 m^2 and 4 m
  // / |d|, and the first has no hit unless its own t is a number.  (A
  // primitive with a NaN coordinate is in no box but its own, so the scene's
  // does not show it: whether such a one is met before a nearer hit is left
  // open.)
  float corner = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float c = fmaxf(fabsf(__ldg(A.root_box + k)), fabsf(__ldg(A.root_box + 3 + k)));
    corner += c * c;
  }
  while (true) {
    unsigned long long first = 0;
    if (lane == 0) first = atomicAdd(A.counter, (unsigned long long)A.lanes);
    first = __shfl_sync(FULL_MASK, first, 0);
    if (first >= A.nrays) break;
    const uint64_t r = first + lane;
    const bool mine = lane < A.lanes && r < A.nrays;
    bool one = false;
    if (mine) {
      Ray R;
      ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
      pool_ray(S, lane, R, 0u, 0u);
      const float mm = R.ox * R.ox + R.oy * R.oy + R.oz * R.oz + corner;
      const float dd = R.dx * R.dx + R.dy * R.dy + R.dz * R.dz;
      if (!(mm * fmaxf(dd, 1.0f) < 1e30f && dd < 1e30f && dd > 1e-30f)) S.best[lane] = kOddKey;
      s_dir[w][lane] = make_float4(R.dx, R.dy, R.dz, 0.0f);
      if (A.n == 1) {
        float tn;
        one = ray_box(R, A.root_box[0], A.root_box[1], A.root_box[2], A.root_box[3], A.root_box[4], A.root_box[5],
                      R.tmax, tn);
      }
    }
    if (!pool_walk<false, V8>(S, A.bvh, mine && A.n > 1, one, prims)) {
      if (lane == 0) atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
      break;
    }
    if (mine) user_hit(A, r, S.best[lane], s_u[w][lane], s_odd[w][lane]);
    __syncwarp();
  }
  if (lane < kPoolRays) user_odds(A, s_odd[w][lane]);
}

}  // namespace gprtcu

using namespace gprtcu;

namespace {

int user_grid(uint64_t n) {
  const uint64_t g = (n + 255) / 256, cap = (uint64_t)gprtcu_num_sms() * 16;
  return (int)(g < cap ? (g ? g : 1) : cap);
}

template <typename PRIMS>
gprtcuStatus trace_user(const gprtcuLbvh *bvh, PRIMS prims, const float *rays, uint64_t nrays, int any, int exit_test,
                        gprtcuHit *hits, float *u, void *scratch, size_t scratch_bytes, cudaStream_t stream) {
  if (!bvh || (!rays && nrays) || (!hits && nrays)) return GPRTCU_ERR_INVALID_ARG;
  if (nrays == 0) return GPRTCU_OK;
  if (bvh->numPrims == 0 || !bvh->ids || !bvh->rootBox || (bvh->numPrims > 1 && !bvh->bvh2))
    return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)rays & 15) || ((uintptr_t)bvh->bvh2 & 15)) return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  if (scratch_bytes < sizeof(ScratchHeader)) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  ScratchHeader *hdr = (ScratchHeader *)scratch;
  unsigned long long *counter = reinterpret_cast<unsigned long long *>(&hdr->ticket[0]);
  GPRTCU_TRY(cudaMemsetAsync(scratch, 0, sizeof(ScratchHeader), stream));
  const bool v8 = ((uintptr_t)bvh->bvh2 & 31) == 0;
  // The pool while it is the faster form: 12/6 chunks per warp, 113,664 rays
  // on 148 SMs, and 16/6, 151,552 rays, for up to 100,000 primitives.  150,001
  // rays, plain walk / pool / lane per ray: 10,001 spheres 144 / 143 / 153 us,
  // 50,001 269 / 250 / 272, 200,001 400 / 409 / 378; 10,001 swept spheres 77 / 81 /
  // 85, 50,001 186 / 172 / 187, 1,000,001 514 / 519 / 474.  Below
  // 16,384 primitives, whose walks are short, it ends at 9/6, 85,248 rays
  // (70,001 on 10,001 swept spheres pool / k_user_lane 50.8 / 54.9 us), below
  // 8,192 at 6/6.  From there up to one ray per lane that fits, and below 2,048
  // for any number, the tests run where they are met (k_user_lane): where
  // primitives lie apart a queue costs more than its full lanes give, and
  // where they overlap this is still faster than a plain walk.  Plain walk /
  // pool or queue / k_user_lane: 113,001 rays on 1,001 spheres 45.1 / 51.2 /
  // 38.9 us, on 5,001 84.4 / 86.9 / 73.9, on as many swept spheres 26.8 / 29.2 /
  // 26.5 and 49.5 / 49.4 / 45.4; 150,001 on 10,001 of them 77.5 / 81.7 / 69.3;
  // 1,000,001 on 101 of them 33.5 / 58.8 / 34.2, on 101 wide ones that overlap
  // 883 / 650 / 759.  From 2,048 on, more rays find the queue faster or level:
  // 1,000,001 on 5,001 spheres that overlap 669 / 435 / 623.
  const uint32_t n = bvh->numPrims;
  const RayGrid few =
      any ? RayGrid{0, 0} : pool_grid(nrays, n < 8192 ? 6 : n < 16384 ? 9 : n <= 100000 ? 16 : 12);
  const bool lane = any || n < 2048 ||
                    (n < 16384 && nrays <= (uint64_t)gprtcu_num_sms() * kUserAnyCtas * kUserThreads);
  const RayGrid g = few.lanes ? few : ray_grid(nrays, lane ? kUserAnyCtas : kUserCtas<PRIMS>, kUserWarps);
  UserArgs<PRIMS> a{(const Bvh2Node *)bvh->bvh2, bvh->ids, bvh->numPrims, bvh->rootBox, prims, exit_test != 0,
                    (const float4 *)rays, nrays, g.lanes, (Hit *)hits, u, counter, &hdr->status};
  auto launch = [&](auto kernel, int threads) { kernel<<<g.ctas, threads, 0, stream>>>(a); };
  if (any) v8 ? launch(k_user_lane<PRIMS, true, true>, kUserThreads) : launch(k_user_lane<PRIMS, true, false>, kUserThreads);
  else if (few.lanes) v8 ? launch(k_user_pool<PRIMS, true>, kPoolThreads) : launch(k_user_pool<PRIMS, false>, kPoolThreads);
  else if (lane) v8 ? launch(k_user_lane<PRIMS, false, true>, kUserThreads) : launch(k_user_lane<PRIMS, false, false>, kUserThreads);
  else v8 ? launch(k_user_closest<PRIMS, true>, kUserThreads) : launch(k_user_closest<PRIMS, false>, kUserThreads);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

}  // namespace

extern "C" GPRTCU_API gprtcuStatus gprtcuSphereBounds(const float *spheres, uint32_t n, float *aabbs,
                                                      gprtcuStream stream) {
  if (n && (!spheres || !aabbs || ((uintptr_t)spheres & 15))) return GPRTCU_ERR_INVALID_ARG;
  if (n == 0) return GPRTCU_OK;
  k_sphere_bounds<<<user_grid(n), 256, 0, (cudaStream_t)stream>>>((const float4 *)spheres, n, aabbs);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuLssBounds(const float *vertices, const uint32_t *indices, uint32_t n,
                                                   int endcap0, int endcap1, float *aabbs, gprtcuStream stream) {
  if (n && (!vertices || !indices || !aabbs || ((uintptr_t)vertices & 15) || ((uintptr_t)indices & 7)))
    return GPRTCU_ERR_INVALID_ARG;
  if (n == 0) return GPRTCU_OK;
  k_lss_bounds<<<user_grid(n), 256, 0, (cudaStream_t)stream>>>((const float4 *)vertices, (const uint2 *)indices, n,
                                                               endcap0, endcap1, aabbs);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuTraceSpheres(const gprtcuLbvh *bvh, const float *spheres, const float *rays,
                                                      uint64_t numRays, int anyHit, int exitTest, gprtcuHit *hits,
                                                      float *hitU, void *scratch, size_t scratchBytes,
                                                      gprtcuStream stream) {
  if (!spheres || ((uintptr_t)spheres & 15)) return GPRTCU_ERR_INVALID_ARG;
  return trace_user(bvh, SpherePrims{(const float4 *)spheres}, rays, numRays, anyHit, exitTest, hits, hitU, scratch,
                    scratchBytes, (cudaStream_t)stream);
}

extern "C" GPRTCU_API gprtcuStatus gprtcuTraceLss(const gprtcuLbvh *bvh, const float *vertices,
                                                  const uint32_t *indices, int endcap0, int endcap1,
                                                  const float *rays, uint64_t numRays, int anyHit, int exitTest,
                                                  gprtcuHit *hits, float *hitU, void *scratch, size_t scratchBytes,
                                                  gprtcuStream stream) {
  if (!vertices || !indices || ((uintptr_t)vertices & 15) || ((uintptr_t)indices & 7)) return GPRTCU_ERR_INVALID_ARG;
  return trace_user(bvh, LssPrims{(const float4 *)vertices, (const uint2 *)indices, endcap0 != 0, endcap1 != 0}, rays,
                    numRays, anyHit, exitTest, hits, hitU, scratch, scratchBytes, (cudaStream_t)stream);
}
