// inst.cu -- two-level instancing: a top-level LBVH over instances of the
// meshes of a bottom-level batch, traced in one kernel.
//
// Instance record: the reference's gprt::Instance (gprt/gprt_shared.h:92-101;
// gprtInstanceAccelCreate, gprt/gprt_host.h:1418): a row-major 3x4
// object-to-world transform, customIndex (24 bits) and mask (8 bits),
// geometryIndex and flags (not used here), and the bottom-level structure --
// here the mesh index in a batched LBVH (gprtcuBatchBuildTriangles), or 0 for
// a single-mesh LBVH.
//
// gprtcuInstancesPrepare computes, per instance, the world-to-object matrix
// (adjugate / determinant in double, fixed operation order, rounded once to
// float) and the world box of the mesh's root box (its eight corners mapped
// in double, rounded outward); the caller builds the top level over those
// boxes with gprtcuLbvhBuildBoxes.  gprtcuTraceInstances walks the top level
// with the world ray; at an instance whose mask meets the ray mask it maps
// the ray into object space (((w0*x + w1*y) + w2*z) + w3 per component, in
// float; tmin/tmax kept: an affine map keeps the ray parameter) and walks
// that mesh's binary LBVH with the same watertight test as the one-level
// traversal.  Closest hit: smallest t, ties to the lowest (instance,
// primitive); t is the refined plane-equation distance in the winning
// instance's object space.
#include "bvh2.cuh"
#include "common.cuh"
#include "lbvh.cuh"
#include "rtmath.cuh"

namespace gprtcu {

struct __align__(16) InstanceRec {
  float m[12];
  uint32_t custom_mask;
  uint32_t geom_flags;
  unsigned long long blas;
};
static_assert(sizeof(InstanceRec) == 64, "64-byte instance record");

__global__ void k_instances_prepare(const InstanceRec *inst, uint32_t n, const float *root_boxes, uint32_t meshes,
                                    float *w2o, float *boxes) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const InstanceRec r = inst[i];
    const double a00 = r.m[0], a01 = r.m[1], a02 = r.m[2], t0 = r.m[3];
    const double a10 = r.m[4], a11 = r.m[5], a12 = r.m[6], t1 = r.m[7];
    const double a20 = r.m[8], a21 = r.m[9], a22 = r.m[10], t2 = r.m[11];
    const double c00 = __dsub_rn(__dmul_rn(a11, a22), __dmul_rn(a12, a21));
    const double c01 = __dsub_rn(__dmul_rn(a12, a20), __dmul_rn(a10, a22));
    const double c02 = __dsub_rn(__dmul_rn(a10, a21), __dmul_rn(a11, a20));
    const double c10 = __dsub_rn(__dmul_rn(a02, a21), __dmul_rn(a01, a22));
    const double c11 = __dsub_rn(__dmul_rn(a00, a22), __dmul_rn(a02, a20));
    const double c12 = __dsub_rn(__dmul_rn(a01, a20), __dmul_rn(a00, a21));
    const double c20 = __dsub_rn(__dmul_rn(a01, a12), __dmul_rn(a02, a11));
    const double c21 = __dsub_rn(__dmul_rn(a02, a10), __dmul_rn(a00, a12));
    const double c22 = __dsub_rn(__dmul_rn(a00, a11), __dmul_rn(a01, a10));
    const double det = __dadd_rn(__dadd_rn(__dmul_rn(a00, c00), __dmul_rn(a01, c01)), __dmul_rn(a02, c02));
    float *w = w2o + 12 * (size_t)i;
    float *bx = boxes + 6 * (size_t)i;
    const uint32_t mesh = (uint32_t)r.blas;
    if (!(det != 0.0) || !isfinite(det) || mesh >= meshes) {
      // never entered: zero matrix, empty box
      for (int k = 0; k < 12; ++k) w[k] = 0.0f;
      for (int k = 0; k < 3; ++k) {
        bx[k] = __int_as_float(0x7f800000);
        bx[3 + k] = __int_as_float(0xff800000);
      }
      continue;
    }
    const double in[9] = {__ddiv_rn(c00, det), __ddiv_rn(c10, det), __ddiv_rn(c20, det),
                          __ddiv_rn(c01, det), __ddiv_rn(c11, det), __ddiv_rn(c21, det),
                          __ddiv_rn(c02, det), __ddiv_rn(c12, det), __ddiv_rn(c22, det)};
    const double tv[3] = {t0, t1, t2};
#pragma unroll
    for (int row = 0; row < 3; ++row) {
      const double u = -__dadd_rn(__dadd_rn(__dmul_rn(in[3 * row], tv[0]), __dmul_rn(in[3 * row + 1], tv[1])),
                                  __dmul_rn(in[3 * row + 2], tv[2]));
      w[4 * row] = __double2float_rn(in[3 * row]);
      w[4 * row + 1] = __double2float_rn(in[3 * row + 1]);
      w[4 * row + 2] = __double2float_rn(in[3 * row + 2]);
      w[4 * row + 3] = __double2float_rn(u);
    }
    // world box of the mesh's root box: eight corners in double, rounded outward
    const float *rb = root_boxes + 6 * (size_t)mesh;
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int c = 0; c < 8; ++c) {
      const double p[3] = {(double)rb[(c & 1) ? 3 : 0], (double)rb[(c & 2) ? 4 : 1], (double)rb[(c & 4) ? 5 : 2]};
      for (int row = 0; row < 3; ++row) {
        const double v = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn((double)r.m[4 * row], p[0]),
                                                       __dmul_rn((double)r.m[4 * row + 1], p[1])),
                                             __dmul_rn((double)r.m[4 * row + 2], p[2])),
                                   (double)r.m[4 * row + 3]);
        lo[row] = fmin(lo[row], v);
        hi[row] = fmax(hi[row], v);
      }
    }
    for (int k = 0; k < 3; ++k) {
      bx[k] = __double2float_rd(lo[k]);
      bx[3 + k] = __double2float_ru(hi[k]);
    }
  }
}

__device__ __forceinline__ void ray_to_object(const float *w, const Ray &W, Ray &O) {
  const float o[3] = {W.ox, W.oy, W.oz}, d[3] = {W.dx, W.dy, W.dz};
  float ro[3], rd[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float w0 = __ldg(w + 4 * i), w1 = __ldg(w + 4 * i + 1), w2 = __ldg(w + 4 * i + 2), w3 = __ldg(w + 4 * i + 3);
    ro[i] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(w0, o[0]), __fmul_rn(w1, o[1])), __fmul_rn(w2, o[2])), w3);
    rd[i] = __fadd_rn(__fadd_rn(__fmul_rn(w0, d[0]), __fmul_rn(w1, d[1])), __fmul_rn(w2, d[2]));
  }
  ray_setup(make_float4(ro[0], ro[1], ro[2], W.tmin), make_float4(rd[0], rd[1], rd[2], W.tmax), O);
}

struct InstArgs {
  const Bvh2Node *tnodes;  // top level
  const uint32_t *tids;
  uint32_t ninst;
  const float *troot;
  const InstanceRec *inst;
  const float *w2o;
  const Bvh2Node *nodes;  // bottom level
  const float4 *leaf;
  const uint32_t *tri_off;  // null: one mesh of n triangles
  uint32_t meshes, n;
  const float4 *rays;
  uint64_t nrays;
  uint32_t ray_mask;
  int lanes;  // rays a warp holds at a time
  Hit *hits;
  uint32_t *hit_inst;
  unsigned long long *counter;
  uint32_t *err;
};

constexpr int kInstThreads = 128;
constexpr int kInstWarps = kInstThreads / 32;
constexpr int kInstShared = 10;  // stack entries in shared memory
constexpr int kInstDepth = 128;  // 62 levels of each tree
constexpr int kInstRefill = 4;
constexpr int kInstSteps = 6;
constexpr int kInstFlush = 12;
constexpr int kInstQueue = 96;  // a step queues at most 64
constexpr int kInstCtas = 8;
constexpr int kWalkLeave = kWalkEnd + 1;  // below a mesh's entries: back to the top level

// Finished rays that hit something, refined 32 at a time.
struct InstRefineQueue {
  unsigned long long ray[64];
  uint32_t inst[64], slot[64];
};

// t of the winner on its object-space ray, recomputed from the ray (the same
// operations, so the same bits as during the walk).
__device__ __forceinline__ void inst_refine(const InstArgs &A, const InstRefineQueue &q, int first, int count) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane < count) {
    const unsigned long long r = q.ray[first + lane];
    const uint32_t inst = q.inst[first + lane], slot = q.slot[first + lane];
    const float4 o = __ldg(A.rays + 2 * r), d = __ldg(A.rays + 2 * r + 1);
    Ray W, O;
    W.ox = o.x; W.oy = o.y; W.oz = o.z; W.tmin = o.w;
    W.dx = d.x; W.dy = d.y; W.dz = d.z; W.tmax = d.w;
    ray_to_object(A.w2o + 12 * (size_t)inst, W, O);
    const float4 a = __ldg(A.leaf + 3 * (size_t)slot), b = __ldg(A.leaf + 3 * (size_t)slot + 1),
                 c = __ldg(A.leaf + 3 * (size_t)slot + 2);
    const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
    Hit h;
    h.prim = __float_as_uint(a.w);
    h.t = refine_t(O, v0, v1, v2);
    A.hits[r] = h;
    if (A.hit_inst) A.hit_inst[r] = inst;
  }
  __syncwarp();
}

// One lane per ray from a global counter.  A lane walks the top level with
// its world ray; the lanes that reach an instance within the same few steps
// map their rays into object space together and walk that mesh on the same
// stack, above a mark that leads back to the top level.  Closest hit queues its
// triangle tests per warp and runs them with all lanes (as the one-level
// traversal does); the queue is emptied before a lane with tests in it enters
// another instance, so the tests of a lane all belong to the instance it
// entered last, whose object-space ray is in shared memory.
// With entries, node steps and tests of single lanes each taking the whole
// warp's time, 7.6 of 32 lanes were active; now 19 are, and the L1 data pipe
// (76 % busy, see load_child) and load latency bound it.  4.2 M rays over
// 16,384 instances: 18.0 -> 10.9 ms; 200,001 rays: 1.39 -> 1.01 ms.  Letting
// entering lanes wait for 2 / 4 / 8 of them: 10.9 / 10.9 / 10.9 ms and 1.04 /
// 1.14 / 1.31 ms (and 0.33 / 0.38 / 0.40 / 0.45 ms for 1 / 2 / 4 / 8 on 200,001
// rays over 1,001 instances, 0.37 before).  8 CTAs per SM instead of 6: 12.1 ->
// 10.8 ms; 2 / 4 / 6 / 8 node steps between two looks at entries, flush and
// refill: 12.5 / 12.1 / 11.2 / 12.0 ms then.  10 stack entries in shared memory
// against 8 and 6: 10.8 / 11.2 / 11.5 ms.  With no more rays to take, a flush
// comes once every lane still walking has a test queued (four at least): over
// few instances a warp's last rays otherwise walk on with a stale culling
// distance.  20,001 rays over 64 instances of 64 / 4 meshes, 400,001 triangles
// together: 101 / 171 -> 84 / 148 us (92 / 163 in the plain walk); with 3,000
// instances as before; 115,001 rays over 200 instances of 4 meshes 367 -> 377 us
// (422).  Six or eight tests at least: 99 / 91 us on the first.
template <bool ANY, bool V8>
__global__ void __launch_bounds__(kInstThreads, kInstCtas) k_trace_inst(const InstArgs A) {
  __shared__ float2 s_stack[kInstShared][kInstThreads];
  __shared__ InstRefineQueue s_rq[kInstWarps];
  __shared__ uint32_t s_qslot[kInstWarps][kInstQueue];
  __shared__ uint8_t s_qlane[kInstWarps][kInstQueue];
  __shared__ unsigned long long s_key[kInstWarps][32];  // closest (t, id) of the tests since the last merge
  __shared__ uint32_t s_kslot[kInstWarps][32];
  __shared__ float s_obj[7][kInstThreads];    // origin, Sx, Sy, Sz; tmax
  __shared__ int s_objk[kInstThreads];        // kx | ky << 2 | kz << 4
  __shared__ uint32_t s_best[2][kInstThreads];  // instance and leaf slot of the best hit
  __shared__ unsigned long long s_rid[kInstThreads];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, wbase = tid & ~31;
  const uint32_t lt = (1u << lane) - 1u;
  InstRefineQueue &rq = s_rq[w];
  uint32_t *qslot = s_qslot[w];
  uint8_t *qlane = s_qlane[w];
  const float kNone = __int_as_float(0x7fffffff);
  bool active = false, drained = false, pending = false, inside = false;
  RayPairs P;
  P.nxy = P.nzz = P.ixy = P.izz = 0;
  P.tmin = 0.0f;
  float bt = 0.0f;
  uint32_t ci = 0, base_leaf = 0, base_node = 0;  // the instance entered last, its mesh's arrays
  int nq = 0, nrq = 0;
  Walk W;
  W.start();
  W.node = kWalkEnd;
  float2 *const sh = &s_stack[0][tid];
  float2 over[kInstDepth - kInstShared];

  // one triangle of lane o's object-space ray
  auto tri_test = [&](uint32_t slot, int o, float tmin, uint32_t &id, float &t) -> bool {
    Ray Q;
    Q.ox = s_obj[0][wbase + o];
    Q.oy = s_obj[1][wbase + o];
    Q.oz = s_obj[2][wbase + o];
    Q.Sx = s_obj[3][wbase + o];
    Q.Sy = s_obj[4][wbase + o];
    Q.Sz = s_obj[5][wbase + o];
    Q.tmax = s_obj[6][wbase + o];
    Q.tmin = tmin;
    const int k = s_objk[wbase + o];
    Q.kx = k & 3;
    Q.ky = (k >> 2) & 3;
    Q.kz = k >> 4;
    const float4 a = __ldg(A.leaf + 3 * (size_t)slot), b = __ldg(A.leaf + 3 * (size_t)slot + 1),
                 c = __ldg(A.leaf + 3 * (size_t)slot + 2);
    const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
    id = __float_as_uint(a.w);
    return isect_tri(Q, v0, v1, v2, t);
  };
  // folds a hit of instance ci into the ray's best (smallest t, then lowest
  // instance, then lowest primitive)
  auto take_hit = [&](float t, uint32_t id, uint32_t slot) {
    const uint32_t bi = s_best[0][tid];
    if (bi == kMiss || t < bt ||
        (t == bt && (ci < bi || (ci == bi && id < __float_as_uint(__ldg(A.leaf + 3 * (size_t)s_best[1][tid]).w))))) {
      s_best[0][tid] = ci;
      s_best[1][tid] = slot;
      bt = t;
    }
  };
  // every queued test by all lanes (warp-uniform call)
  auto flush = [&]() {
    __syncwarp();
    for (int b = 0; b < nq; b += 32) {
      const int e = b + lane;
      const bool on = e < nq;
      const uint32_t slot = on ? qslot[e] : 0u;
      const int o = on ? qlane[e] : lane;
      const float tmin = __shfl_sync(FULL_MASK, P.tmin, o);
      unsigned long long key = ~0ull;
      uint32_t id;
      float t;
      if (on && tri_test(slot, o, tmin, id, t)) {
        key = ((unsigned long long)t_order(t) << 32) | id;
        atomicMin(&s_key[w][o], key);
      }
      __syncwarp();
      if (key != ~0ull && s_key[w][o] == key) s_kslot[w][o] = slot;  // one winner per owner
      __syncwarp();
    }
    if (pending) {
      const unsigned long long key = s_key[w][lane];
      if (key != ~0ull) {
        take_hit(t_from_order((uint32_t)(key >> 32)), (uint32_t)key, s_kslot[w][lane]);
        s_key[w][lane] = ~0ull;
      }
      pending = false;
    }
    nq = 0;
    __syncwarp();
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
      if (warp_take(active, drained, A.lanes, kInstRefill, A.nrays, A.counter, r)) {
        Ray R;
        ray_setup(__ldg(A.rays + 2 * r), __ldg(A.rays + 2 * r + 1), R);
        active = true;
        inside = false;
        P = ray_pairs(R);
        bt = R.tmax;
        W.start();
        s_obj[6][tid] = R.tmax;
        s_best[0][tid] = kMiss;
        s_key[w][lane] = ~0ull;
        s_rid[tid] = r;
        if (A.ninst == 1) {
          float tn;
          W.node = ~0;  // the single instance is the root leaf
          W.t = R.tmin;
          if (!ray_box(R, A.troot[0], A.troot[1], A.troot[2], A.troot[3], A.troot[4], A.troot[5], bt, tn))
            W.node = kWalkEnd;
        }
      }
    }
    if (!__any_sync(FULL_MASK, active)) {
      if (drained) break;
      continue;
    }
#pragma unroll 1
    for (int step = 0; step < kInstSteps; ++step) {
      const bool on = W.node >= 0;
      float t0 = kNone, t1 = kNone;
      int r0 = 0, r1 = 0;
      bool leaf0 = false, leaf1 = false, found = false;
      if (on && W.t <= bt) {
        const Bvh2Node *nd = inside ? A.nodes + base_node + W.node : A.tnodes + W.node;
        const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
        t0 = child_entry(c0, P, bt);
        t1 = child_entry(c1, P, bt);
        r0 = c0.ref;
        r1 = c1.ref;
        leaf0 = inside && r0 < 0 && t0 == t0;
        leaf1 = inside && r1 < 0 && t1 == t1;
        if (ANY) {
          uint32_t id;
          float t;
          if (leaf0 && tri_test(base_leaf + (uint32_t)~r0, lane, P.tmin, id, t))
            take_hit(t, id, base_leaf + (uint32_t)~r0);
          if (leaf1 && t1 <= bt && tri_test(base_leaf + (uint32_t)~r1, lane, P.tmin, id, t))
            take_hit(t, id, base_leaf + (uint32_t)~r1);
          found = (leaf0 || leaf1) && s_best[0][tid] != kMiss;
        }
        if (leaf0) t0 = kNone;
        if (leaf1) t1 = kNone;
      }
      if (!walk_next<kInstThreads, kInstShared, kInstDepth>(W, sh, over, on, t0, r0, t1, r1)) {
        atomicCAS(A.err, 0u, 5u);  // traversal stack overflow
        W.node = kWalkEnd;
      }
      if (ANY && found) W.node = kWalkEnd;
      if (W.node == kWalkLeave) {  // back to the world ray; the next step pops
        inside = false;
        const unsigned long long r = s_rid[tid];
        const float4 o = __ldg(A.rays + 2 * r), d = __ldg(A.rays + 2 * r + 1);
        const float iz = __frcp_rn(d.z);
        P.nxy = pk2(-o.x, -o.y);
        P.nzz = pk2(-o.z, -o.z);
        P.ixy = pk2(__frcp_rn(d.x), __frcp_rn(d.y));
        P.izz = pk2(iz, iz);
        W.node = 0;
        W.t = kNone;
      }
      if (!ANY && __any_sync(FULL_MASK, leaf0 || leaf1)) {
        if (nq > kInstQueue - 64) flush();
        queue(leaf0, base_leaf + (uint32_t)~r0);
        queue(leaf1, base_leaf + (uint32_t)~r1);
      }
    }
    // ---- instances: enter them together
    const unsigned entering = __ballot_sync(FULL_MASK, W.node < 0 && W.node > kWalkLeave);
    if (entering) {
      const bool enter = W.node < 0 && W.node > kWalkLeave;
      if (!ANY && __any_sync(FULL_MASK, enter && pending)) flush();
      if (!ANY && nq > kInstQueue - 32) flush();
      bool one = false, found = false;
      if (enter) {
        const uint32_t ti = __ldg(A.tids + (uint32_t)~W.node);
        W.node = 0;  // the next step pops, unless the instance is entered below
        const float t = W.t;
        W.t = kNone;
        const uint32_t cm = __ldg(&A.inst[ti].custom_mask);
        const uint32_t mesh = (uint32_t)__ldg(&A.inst[ti].blas);
        const float *wm = A.w2o + 12 * (size_t)ti;
        if (t <= bt && ((cm >> 24) & A.ray_mask) && mesh < A.meshes &&
            (__ldg(wm) != 0.0f || __ldg(wm + 1) != 0.0f || __ldg(wm + 2) != 0.0f)) {  // singular: all zero
          const unsigned long long r = s_rid[tid];
          const float4 o4 = __ldg(A.rays + 2 * r), d4 = __ldg(A.rays + 2 * r + 1);
          Ray R, O;
          R.ox = o4.x; R.oy = o4.y; R.oz = o4.z; R.tmin = o4.w;
          R.dx = d4.x; R.dy = d4.y; R.dz = d4.z; R.tmax = d4.w;
          ray_to_object(wm, R, O);
          ci = ti;
          base_leaf = A.tri_off ? __ldg(A.tri_off + mesh) : 0u;
          const uint32_t cnt = A.tri_off ? __ldg(A.tri_off + mesh + 1) - base_leaf : A.n;
          base_node = base_leaf - mesh;
          s_obj[0][tid] = O.ox;
          s_obj[1][tid] = O.oy;
          s_obj[2][tid] = O.oz;
          s_obj[3][tid] = O.Sx;
          s_obj[4][tid] = O.Sy;
          s_obj[5][tid] = O.Sz;
          s_objk[tid] = O.kx | (O.ky << 2) | (O.kz << 4);
          if (cnt == 1) {
            const float4 a = __ldg(A.leaf + 3 * (size_t)base_leaf), b = __ldg(A.leaf + 3 * (size_t)base_leaf + 1),
                         c = __ldg(A.leaf + 3 * (size_t)base_leaf + 2);
            float tn;
            one = ray_box(O, fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z)),
                          fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z)), bt,
                          tn) &&
                  tn <= bt;
            if (ANY && one) {
              uint32_t id;
              float th;
              if (tri_test(base_leaf, lane, P.tmin, id, th)) {
                take_hit(th, id, base_leaf);
                found = true;
              }
            }
          } else {
            P = ray_pairs(O);
            inside = true;
            W.t = t;
            if (!walk_push<kInstThreads, kInstShared, kInstDepth>(W, sh, over, kWalkLeave, 0.0f)) {
              atomicCAS(A.err, 0u, 5u);
              W.node = kWalkEnd;
            }
          }
        }
      }
      if (ANY) {
        if (found) W.node = kWalkEnd;
      } else {
        __syncwarp();
        queue(one, base_leaf);
      }
    }
    const bool done = W.node == kWalkEnd;
    if (!ANY) {
      const unsigned waiting = __ballot_sync(FULL_MASK, done && active && pending);
      const unsigned running = __ballot_sync(FULL_MASK, active && !done);
      if (nq >= kInstFlush || (drained && nq >= max(__popc(running), 4)) || (waiting && (!running || A.lanes - __popc(running) >= kInstRefill))) flush();
    }
    const bool fin = active && done && !pending;
    if (__any_sync(FULL_MASK, fin)) {
      const bool hit = fin && s_best[0][tid] != kMiss;
      if (fin && !hit) {
        const unsigned long long r = s_rid[tid];
        Hit h;
        h.prim = kMiss;
        h.t = __int_as_float(0x7f800000);
        A.hits[r] = h;
        if (A.hit_inst) A.hit_inst[r] = kMiss;
      }
      const unsigned m = __ballot_sync(FULL_MASK, hit);
      if (hit) {
        const int k = nrq + __popc(m & lt);
        rq.ray[k] = s_rid[tid];
        rq.inst[k] = s_best[0][tid];
        rq.slot[k] = s_best[1][tid];
      }
      nrq += __popc(m);
      if (nrq >= 32) {
        nrq -= 32;
        inst_refine(A, rq, nrq, 32);
      }
      if (fin) active = false;
    }
  }
  inst_refine(A, rq, 0, nrq);
}

}  // namespace gprtcu

using namespace gprtcu;

extern "C" GPRTCU_API gprtcuStatus gprtcuInstancesPrepare(const gprtcuInstance *instances, uint32_t numInstances,
                                                          const float *blasRootBoxes, uint32_t numMeshes,
                                                          float *worldToObject, float *worldBoxes,
                                                          gprtcuStream stream) {
  if (numInstances == 0) return GPRTCU_OK;
  if (!instances || !blasRootBoxes || !worldToObject || !worldBoxes || numMeshes == 0) return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)instances & 15)) return GPRTCU_ERR_INVALID_ARG;
  const uint64_t g = (numInstances + 255) / 256, cap = (uint64_t)gprtcu_num_sms() * 16;
  k_instances_prepare<<<(unsigned)(g < cap ? g : cap), 256, 0, (cudaStream_t)stream>>>(
      (const InstanceRec *)instances, numInstances, blasRootBoxes, numMeshes, worldToObject, worldBoxes);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuTraceInstances(const gprtcuLbvh *tlas, const gprtcuInstance *instances,
                                                        const float *worldToObject, const gprtcuLbvh *blas,
                                                        const uint32_t *triOffsets, uint32_t numMeshes,
                                                        const float *rays, uint64_t numRays, uint32_t rayMask,
                                                        int anyHit, gprtcuHit *hits, uint32_t *hitInstance,
                                                        void *scratch, size_t scratchBytes, gprtcuStream stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!tlas || !instances || !worldToObject || !blas || numMeshes == 0 || (numMeshes > 1 && !triOffsets))
    return GPRTCU_ERR_INVALID_ARG;
  if ((!rays || !hits) && numRays) return GPRTCU_ERR_INVALID_ARG;
  if (numRays == 0) return GPRTCU_OK;
  if (tlas->numPrims == 0 || !tlas->ids || !tlas->rootBox || (tlas->numPrims > 1 && !tlas->bvh2))
    return GPRTCU_ERR_INVALID_ARG;
  if (blas->numPrims == 0 || !blas->leafTris || (blas->numPrims > numMeshes && !blas->bvh2)) return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)rays & 15) || ((uintptr_t)instances & 15) || ((uintptr_t)tlas->bvh2 & 15) ||
      ((uintptr_t)blas->bvh2 & 15) || ((uintptr_t)blas->leafTris & 15))
    return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  if (scratchBytes < sizeof(ScratchHeader)) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  ScratchHeader *hdr = (ScratchHeader *)scratch;
  unsigned long long *counter = reinterpret_cast<unsigned long long *>(&hdr->ticket[0]);
  GPRTCU_TRY(cudaMemsetAsync(scratch, 0, sizeof(ScratchHeader), stream));
  const RayGrid g = ray_grid(numRays, kInstCtas, kInstWarps, 8);
  InstArgs a;
  a.tnodes = (const Bvh2Node *)tlas->bvh2;
  a.tids = tlas->ids;
  a.ninst = tlas->numPrims;
  a.troot = tlas->rootBox;
  a.inst = (const InstanceRec *)instances;
  a.w2o = worldToObject;
  a.nodes = (const Bvh2Node *)blas->bvh2;
  a.leaf = (const float4 *)blas->leafTris;
  a.tri_off = numMeshes > 1 ? triOffsets : nullptr;
  a.meshes = numMeshes;
  a.n = blas->numPrims;
  a.rays = (const float4 *)rays;
  a.nrays = numRays;
  a.ray_mask = rayMask;
  a.lanes = g.lanes;
  a.hits = (Hit *)hits;
  a.hit_inst = hitInstance;
  a.counter = counter;
  a.err = &hdr->status;
  auto launch = [&](auto kernel) { kernel<<<g.ctas, kInstThreads, 0, stream>>>(a); };
  const bool v8 = (((uintptr_t)tlas->bvh2 | (uintptr_t)blas->bvh2) & 31) == 0;
  if (anyHit) v8 ? launch(k_trace_inst<true, true>) : launch(k_trace_inst<true, false>);
  else v8 ? launch(k_trace_inst<false, true>) : launch(k_trace_inst<false, false>);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}
