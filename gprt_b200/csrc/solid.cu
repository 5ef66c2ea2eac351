// solid.cu -- solid cells (tetrahedra, pyramids, wedges, hexahedra and
// tetrahedral pairs: the linear finite elements of volume meshes) as
// software-BVH primitives: their bounds, and point location over an LBVH
// built on those bounds (gprtcuLbvhBuildBoxes).
//
// The reference builds a hardware AABB structure over the boxes of its
// SolidBounds compute program (gprt/gprt_fallbacks.slang:467-502) and answers
// TracePoint (gprt/gprt_builtins.slang:80-90: a zero-length ray from the
// point) with SolidIntersection (:504-566), which inverts the cell's
// isoparametric map by Newton's method (intersectPointSolid, :409-464).  Here
// the same arithmetic runs in CUDA with every float operation an explicit
// round-to-nearest intrinsic in the reference's evaluation order, and the
// derivatives the reference takes with forward-mode automatic differentiation
// (fwd_diff of IsoToSupport, :437-439) are written out per cell type with the
// terms that the rules (d(c - a) = -da, d(a b) = da b + a db) make zero left
// out, so the containing cell, its (r, s, t) and its interpolated density are
// bit-identical to the reference's code compiled for the host.
//
// A point lies in a cell's box when lo <= p <= hi on every axis (a zero-length
// ray meets a box exactly then).  Of the cells whose box and Newton inversion
// contain the point, the lowest-numbered one is reported (every hit of a
// point query is at t = 0; ties go to the lowest id, as for rays).
#include "bvh2.cuh"
#include "common.cuh"
#include "lbvh.cuh"

#include <type_traits>

namespace gprtcu {

// Cell types (gprt/gprt_host.h:291-298) and their vertex counts and hit kinds
// (gprt/gprt_fallbacks.slang:289-318).  A tetrahedral pair has eight nodes,
// is evaluated as a trilinear cell and reports the tetrahedron kind.
__device__ __forceinline__ int solid_nodes(uint32_t type) {
  return type == 10u ? 4 : type == 14u ? 5 : type == 13u ? 6 : (type == 12u || type == 23u) ? 8 : 0;
}
__device__ __forceinline__ uint32_t solid_kind(uint32_t type) {
  return type == 23u ? 10u : (type == 10u || type == 12u || type == 13u || type == 14u) ? type : 0u;
}

// Where a cell's data lives: vertex k of the mesh at vertices + k *
// vertexStride (float4 {x, y, z, density}), cell c's vertex indices at
// indices + c * indexStride (uint32 each), its type at types + c * typeStride.
struct SolidView {
  const unsigned char *verts, *idx, *types;
  uint32_t vstride, istride, tstride, n;
  __device__ __forceinline__ uint32_t type(uint32_t c) const { return __ldg(types + (size_t)c * tstride); }
  __device__ __forceinline__ uint32_t index(uint32_t c, int i) const {
    return __ldg(reinterpret_cast<const uint32_t *>(idx + (size_t)c * istride) + i);
  }
  __device__ __forceinline__ float4 vertex(uint32_t k) const {
    return __ldg(reinterpret_cast<const float4 *>(verts + (size_t)k * vstride));
  }
};

// IsoToSupport (gprt/gprt_fallbacks.slang:370-406): the shape functions w of an
// N-node cell at (r, s, t) and their derivatives d[dir], in the reference's
// operation order.  Forward-mode differentiation along one axis gives each
// derivative as a product plus products with a zero derivative; those zeros
// are dropped here.  What is left rounds the same: x + (+-0) is x, and where a
// derivative itself is a zero its sign is lost in the sum over the nodes,
// which starts at +0.  (An infinite r, s or t makes the sums NaN there and
// infinite or NaN here; either way the residual never falls below its bound
// again and the cell is not hit.)  Entries of d that are always zero are not
// read (node_deriv).
template <int N> struct Shape {
  float w[N];
  float dr[N], ds[N], dt[N];
};
template <int N> __device__ __forceinline__ void iso_support(float r, float s, float t, Shape<N> &S) {
  const float mr = __fsub_rn(1.0f, r), ms = __fsub_rn(1.0f, s), mt = __fsub_rn(1.0f, t);
  if constexpr (N == 4) {
    S.w[0] = __fsub_rn(1.0f, __fadd_rn(__fadd_rn(r, s), t));
    S.w[1] = r;
    S.w[2] = s;
    S.w[3] = t;
    S.dr[0] = S.ds[0] = S.dt[0] = -1.0f;
    S.dr[1] = S.ds[2] = S.dt[3] = 1.0f;
    S.dr[2] = S.dr[3] = S.ds[1] = S.ds[3] = S.dt[1] = S.dt[2] = 0.0f;
  } else if constexpr (N == 6) {
    const float rs = __fsub_rn(mr, s);
    S.w[0] = __fmul_rn(rs, mt);
    S.w[1] = __fmul_rn(r, mt);
    S.w[2] = __fmul_rn(s, mt);
    S.w[3] = __fmul_rn(rs, t);
    S.w[4] = __fmul_rn(r, t);
    S.w[5] = __fmul_rn(s, t);
    S.dr[0] = S.ds[0] = -mt;
    S.dr[1] = S.ds[2] = mt;
    S.dr[3] = S.ds[3] = -t;
    S.dr[4] = S.ds[5] = t;
    S.dr[2] = S.dr[5] = S.ds[1] = S.ds[4] = 0.0f;
    S.dt[0] = -rs;
    S.dt[1] = -r;
    S.dt[2] = -s;
    S.dt[3] = rs;
    S.dt[4] = r;
    S.dt[5] = s;
  } else {
    const float a0 = __fmul_rn(mr, ms), a1 = __fmul_rn(r, ms), a2 = __fmul_rn(r, s), a3 = __fmul_rn(mr, s);
    S.w[0] = __fmul_rn(a0, mt);
    S.w[1] = __fmul_rn(a1, mt);
    S.w[2] = __fmul_rn(a2, mt);
    S.w[3] = __fmul_rn(a3, mt);
    S.dr[1] = __fmul_rn(ms, mt);
    S.dr[0] = -S.dr[1];
    S.dr[2] = __fmul_rn(s, mt);
    S.dr[3] = -S.dr[2];
    S.ds[3] = __fmul_rn(mr, mt);
    S.ds[0] = -S.ds[3];
    S.ds[2] = __fmul_rn(r, mt);
    S.ds[1] = -S.ds[2];
    S.dt[0] = -a0;
    S.dt[1] = -a1;
    S.dt[2] = -a2;
    S.dt[3] = -a3;
    if constexpr (N == 5) {
      S.w[4] = t;
      S.dr[4] = S.ds[4] = 0.0f;
      S.dt[4] = 1.0f;
    } else {
      S.w[4] = __fmul_rn(a0, t);
      S.w[5] = __fmul_rn(a1, t);
      S.w[6] = __fmul_rn(a2, t);
      S.w[7] = __fmul_rn(a3, t);
      S.dr[5] = __fmul_rn(ms, t);
      S.dr[4] = -S.dr[5];
      S.dr[6] = __fmul_rn(s, t);
      S.dr[7] = -S.dr[6];
      S.ds[7] = __fmul_rn(mr, t);
      S.ds[4] = -S.ds[7];
      S.ds[6] = __fmul_rn(r, t);
      S.ds[5] = -S.ds[6];
      S.dt[4] = a0;
      S.dt[5] = a1;
      S.dt[6] = a2;
      S.dt[7] = a3;
    }
  }
}
// Whether node i's shape function varies along axis dir at all.
template <int N> __device__ constexpr bool node_deriv(int i, int dir) {
  return N == 4 ? (i == 0 || i == dir + 1)
         : N == 5 ? (i < 4 || dir == 2)
         : N == 6 ? (dir == 2 || i % 3 == 0 || i % 3 == dir + 1)
                  : true;
}

// Determinant of the 3x3 matrix with rows a, b, c (cofactors of the first row).
__device__ __forceinline__ float det3(float a0, float a1, float a2, float b0, float b1, float b2, float c0, float c1,
                                      float c2) {
  const float m0 = __fsub_rn(__fmul_rn(b1, c2), __fmul_rn(b2, c1));
  const float m1 = __fsub_rn(__fmul_rn(b0, c2), __fmul_rn(b2, c0));
  const float m2 = __fsub_rn(__fmul_rn(b0, c1), __fmul_rn(b1, c0));
  return __fadd_rn(__fsub_rn(__fmul_rn(a0, m0), __fmul_rn(a1, m1)), __fmul_rn(a2, m2));
}

// intersectPointSolid (gprt/gprt_fallbacks.slang:409-464): at most five
// Newton steps from GetInitialRST (:320-325); each step uses the residual
// and Jacobian at the current (r, s, t), updates by Cramer's rule, then stops
// if that residual was below 1e-3 on every axis; a Jacobian determinant below
// 1e-20 in magnitude ends the test.  Containment per IsoIsContained
// (:327-340); the density applies the last evaluated shape functions to the
// nodal densities.  q: the cell's N nodes.  (The reference's sums run over
// eight nodes, the absent ones adding zeros.)
template <int N>
__device__ __forceinline__ bool solid_intersect(float px, float py, float pz, const float4 (&q)[N], float4 &rstw) {
  float r = 0.5f, s = 0.5f, t = 0.5f;
  if (N == 4) r = s = t = 0.25f;
  if (N == 5) t = 0.2f;
  float dens = 0.0f;
  bool converged = false;
#pragma unroll 1
  for (int it = 0; it < 5; ++it) {
    Shape<N> S;
    iso_support<N>(r, s, t, S);
    float fx = -px, fy = -py, fz = -pz;
    dens = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      fx = __fadd_rn(fx, __fmul_rn(q[i].x, S.w[i]));
      fy = __fadd_rn(fy, __fmul_rn(q[i].y, S.w[i]));
      fz = __fadd_rn(fz, __fmul_rn(q[i].z, S.w[i]));
      dens = __fadd_rn(dens, __fmul_rn(q[i].w, S.w[i]));
    }
    float c[3][3];
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      float cx = 0.0f, cy = 0.0f, cz = 0.0f;
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (node_deriv<N>(i, dir)) {
          const float d = dir == 0 ? S.dr[i] : (dir == 1 ? S.ds[i] : S.dt[i]);
          cx = __fadd_rn(cx, __fmul_rn(q[i].x, d));
          cy = __fadd_rn(cy, __fmul_rn(q[i].y, d));
          cz = __fadd_rn(cz, __fmul_rn(q[i].z, d));
        }
      c[dir][0] = cx;
      c[dir][1] = cy;
      c[dir][2] = cz;
    }
    const float d = det3(c[0][0], c[0][1], c[0][2], c[1][0], c[1][1], c[1][2], c[2][0], c[2][1], c[2][2]);
    if (fabsf(d) < 1e-20f) return false;
    const float dinv = __fdiv_rn(1.0f, d);
    const float ur = det3(fx, fy, fz, c[1][0], c[1][1], c[1][2], c[2][0], c[2][1], c[2][2]);
    const float us = det3(c[0][0], c[0][1], c[0][2], fx, fy, fz, c[2][0], c[2][1], c[2][2]);
    const float ut = det3(c[0][0], c[0][1], c[0][2], c[1][0], c[1][1], c[1][2], fx, fy, fz);
    r = __fsub_rn(r, __fmul_rn(ur, dinv));
    s = __fsub_rn(s, __fmul_rn(us, dinv));
    t = __fsub_rn(t, __fmul_rn(ut, dinv));
    if (fabsf(fx) < 1e-3f && fabsf(fy) < 1e-3f && fabsf(fz) < 1e-3f) {
      converged = true;
      break;
    }
  }
  if (!converged) return false;
  bool in = r >= 0.0f && s >= 0.0f && t >= 0.0f && r <= 1.0f && s <= 1.0f && t <= 1.0f;
  if (N == 4) in = in && __fadd_rn(__fadd_rn(r, s), t) <= 1.0f;
  if (N == 6) in = in && __fadd_rn(r, s) <= 1.0f;
  if (!in) return false;
  rstw = make_float4(r, s, t, dens);
  return true;
}

// SolidBounds (gprt/gprt_fallbacks.slang:467-502): min / max of the cell's
// vertices and of their densities.  aabbs (optional): two float4 per cell in
// the reference's layout {lo.xyz, hi.x}, {hi.yz, density min, density max};
// boxes (optional): float[6] {lo.xyz, hi.xyz} per cell for the box LBVH.  A
// cell of unknown type has no vertices and an empty box (lo = +FLT_MAX,
// hi = -FLT_MAX), which no point lies in.
__global__ void k_solid_bounds(SolidView sv, float4 *aabbs, float *boxes) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < sv.n; c += gridDim.x * blockDim.x) {
    const int n = solid_nodes(sv.type(c));
    float lx = 3.402823466e38f, ly = 3.402823466e38f, lz = 3.402823466e38f;
    float hx = -3.402823466e38f, hy = -3.402823466e38f, hz = -3.402823466e38f;
    float dlo = 3.402823466e38f, dhi = -3.402823466e38f;
    for (int i = 0; i < n; ++i) {
      const float4 v = sv.vertex(sv.index(c, i));
      lx = fminf(lx, v.x);
      ly = fminf(ly, v.y);
      lz = fminf(lz, v.z);
      hx = fmaxf(hx, v.x);
      hy = fmaxf(hy, v.y);
      hz = fmaxf(hz, v.z);
      dlo = fminf(dlo, v.w);
      dhi = fmaxf(dhi, v.w);
    }
    if (aabbs) {
      aabbs[2 * (size_t)c] = make_float4(lx, ly, lz, hx);
      aabbs[2 * (size_t)c + 1] = make_float4(hy, hz, dlo, dhi);
    }
    if (boxes) {
      float *b = boxes + 6 * (size_t)c;
      b[0] = lx;
      b[1] = ly;
      b[2] = lz;
      b[3] = hx;
      b[4] = hy;
      b[5] = hz;
    }
  }
}

constexpr int kLocateThreads = 128;
constexpr int kLocateWarps = kLocateThreads / 32;
constexpr int kLocateCtas = 6;
constexpr int kLocateShared = 8;  // stack entries in shared memory
constexpr int kLocateStack = 64;
constexpr int kLocateRefill = 4;
constexpr int kLocateSteps = 2;
constexpr int kLocateQueue = 64 + 64 * kLocateSteps;  // leaves met, not looked at yet
constexpr int kLocateBin = 64;    // candidate cells of one node count
constexpr int kLocateChunk = 64;  // points a warp takes at a time
constexpr uint32_t kNoCell = 0xFFFFFFFFu;

struct LocateArgs {
  const Bvh2Node *bvh;
  const uint32_t *ids;
  uint32_t nleaves;
  const float *root_box;
  SolidView sv;
  const float4 *points;
  uint64_t npts;
  int chunk;  // points a warp takes at a time (1 .. kLocateChunk)
  uint2 *hits;
  float4 *rstw;
  unsigned long long *counter;
  uint32_t *err;
};

__device__ __forceinline__ bool point_in(float px, float py, float pz, float lx, float ly, float lz, float hx, float hy,
                                         float hz) {
  return lx <= px && px <= hx && ly <= py && py <= hy && lz <= pz && pz <= hz;
}
__device__ __forceinline__ bool point_in(float px, float py, float pz, const ChildPairs &c) {
  float lx, ly, lz, hx, hy, hz;
  up2(c.b[0], lx, ly);
  up2(c.b[1], hx, hy);
  up2(c.b[2], lz, hz);
  return point_in(px, py, pz, lx, ly, lz, hx, hy, hz);
}

// The first N vertex indices of a cell; I16: records on 16-byte boundaries
// (the default stride), read in 16- and 8-byte loads.
template <int N, bool I16>
__device__ __forceinline__ void cell_indices(const SolidView &sv, uint32_t id, uint32_t (&k)[N]) {
  if constexpr (I16) {
    const unsigned char *p = sv.idx + (size_t)id * sv.istride;
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(p));
    k[0] = a.x;
    k[1] = a.y;
    k[2] = a.z;
    k[3] = a.w;
    if constexpr (N == 5) k[4] = __ldg(reinterpret_cast<const uint32_t *>(p) + 4);
    if constexpr (N == 6) {
      const uint2 b = __ldg(reinterpret_cast<const uint2 *>(p) + 2);
      k[4] = b.x;
      k[5] = b.y;
    }
    if constexpr (N == 8) {
      const uint4 b = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
      k[4] = b.x;
      k[5] = b.y;
      k[6] = b.z;
      k[7] = b.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) k[i] = sv.index(id, i);
  }
}

template <int N, bool I16>
__device__ __forceinline__ bool locate_cell(const SolidView &sv, uint32_t id, float px, float py, float pz,
                                            float4 &r) {
  uint32_t k[N];
  cell_indices<N, I16>(sv, id, k);
  float4 q[N];
#pragma unroll
  for (int i = 0; i < N; ++i) q[i] = sv.vertex(k[i]);
  return solid_intersect<N>(px, py, pz, q, r);
}

// Point location over the box LBVH (gprtcuLbvh.bvh2 over the cells' boxes;
// leaf slot k holds cell ids[k]).  A warp takes a chunk of points; its lanes
// walk one point each and take the chunk's next ones as they finish.  The
// walk only collects leaves whose box holds the point, as (slot, point) in a
// queue per warp.  32 of them at a time are looked up by all lanes and sorted
// by the cell's node count into four bins, and a bin that holds 32 candidates
// runs their Newton inversions, every lane one, whoever's point it is: the
// lanes then run the same shape functions, written for that node count (with
// the types mixed in a warp each inversion ran the code of every type in it,
// and the general code carried all eight nodes and the zero derivatives).  A
// cell that holds the point lowers its owner's best cell with a shared-memory
// atomicMin and leaves its (r, s, t, density) there; candidates at or above
// the owner's best so far are dropped.  When the chunk is walked the rest runs
// in batches that are not full.  4,194,301 points in 2.8 M cells of five
// types: 3.45 -> 2.27 ms, half the instructions; the random node, index and
// vertex fetches (half of them miss L2) at 24 warps per SM bound it now.  5 /
// 6 / 7 CTAs per SM: 2.53 / 2.30 / 2.51 ms (7 spill); chunks of 48 / 64 / 96
// points: 2.35 / 2.30 / 2.27 ms; refill at 8 / 4 idle lanes: 2.30 / 2.27 ms.
// Lanes that wait for their own point's candidates instead of taking the
// next point: 4.3 ms (their candidates then run in batches that are not
// full).  hits: {cell, kind} per point (cell 0xFFFFFFFF, kind 0 when no cell
// holds it); rstw (optional): (r, s, t, density), zero on a miss.
template <bool V8, bool I16>
__global__ void __launch_bounds__(kLocateThreads, kLocateCtas) k_locate_solids(const LocateArgs A) {
  __shared__ int s_stack[kLocateShared][kLocateThreads];
  __shared__ uint32_t s_qslot[kLocateWarps][kLocateQueue];
  __shared__ uint8_t s_qown[kLocateWarps][kLocateQueue];
  __shared__ uint32_t s_bcell[kLocateWarps][4][kLocateBin];
  __shared__ uint8_t s_bown[kLocateWarps][4][kLocateBin];
  __shared__ float s_pt[kLocateWarps][3][kLocateChunk];
  __shared__ uint32_t s_best[kLocateWarps][kLocateChunk];
  __shared__ float4 s_rst[kLocateWarps][kLocateChunk];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t *qslot = s_qslot[w];
  uint8_t *qown = s_qown[w];
  float px = 0.f, py = 0.f, pz = 0.f;
  int point = 0, node = -1, top = -1, sp = 0;  // the lane's walk
  int qn = 0, bn[4] = {0, 0, 0, 0};  // queued leaves, candidates per bin: the same on every lane
  int *const sh = &s_stack[0][tid];
  int over[kLocateStack - kLocateShared];

  auto invert = [&](auto nodes, int bin, int &n) {  // the last up to 32 candidates of a bin
    constexpr int N = decltype(nodes)::value;
    const int count = n < 32 ? n : 32;
    n -= count;
    __syncwarp();
    int own = 0;
    uint32_t id = kNoCell;
    bool in = false;
    float4 r;
    if (lane < count) {
      id = s_bcell[w][bin][n + lane];
      own = s_bown[w][bin][n + lane];
      in = id < *reinterpret_cast<volatile uint32_t *>(&s_best[w][own]) &&
           locate_cell<N, I16>(A.sv, id, s_pt[w][0][own], s_pt[w][1][own], s_pt[w][2][own], r);
      if (in) atomicMin(&s_best[w][own], id);
    }
    __syncwarp();
    if (in && s_best[w][own] == id) s_rst[w][own] = r;  // one winner per owner
    __syncwarp();
  };
  auto run_bin = [&](int bin) {
    if (bin == 0) invert(std::integral_constant<int, 4>(), 0, bn[0]);
    else if (bin == 1) invert(std::integral_constant<int, 5>(), 1, bn[1]);
    else if (bin == 2) invert(std::integral_constant<int, 6>(), 2, bn[2]);
    else invert(std::integral_constant<int, 8>(), 3, bn[3]);
  };
  auto classify = [&]() {  // the last up to 32 queued leaves into the bins
    const int count = qn < 32 ? qn : 32;
    qn -= count;
    __syncwarp();
    uint32_t id = kNoCell;
    int own = 0, n = 0;
    if (lane < count) {
      own = qown[qn + lane];
      id = __ldg(A.ids + qslot[qn + lane]);
      if (id < s_best[w][own]) n = solid_nodes(A.sv.type(id));
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const bool mine = n == (b == 3 ? 8 : b + 4);
      const unsigned m = __ballot_sync(FULL_MASK, mine);
      if (mine) {
        const int k = bn[b] + __popc(m & lt);
        s_bcell[w][b][k] = id;
        s_bown[w][b][k] = (uint8_t)own;
      }
      bn[b] += __popc(m);
    }
    __syncwarp();
  };
  auto queue = [&](bool leaf, uint32_t slot) {
    const unsigned m = __ballot_sync(FULL_MASK, leaf);
    if (leaf) {
      const int k = qn + __popc(m & lt);
      qslot[k] = slot;
      qown[k] = (uint8_t)point;
    }
    qn += __popc(m);
  };

  while (true) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(A.counter, (unsigned long long)A.chunk);
    base = __shfl_sync(FULL_MASK, base, 0);
    if (base >= A.npts) break;
    const int count = (int)min((unsigned long long)A.chunk, A.npts - base);
    for (int i = lane; i < count; i += 32) {
      const float4 p = __ldg(A.points + base + i);
      s_pt[w][0][i] = p.x;
      s_pt[w][1][i] = p.y;
      s_pt[w][2][i] = p.z;
      s_best[w][i] = kNoCell;
    }
    __syncwarp();
    int next = 0;  // the chunk's points up to here are walked or being walked
    while (true) {
      const unsigned idle = __ballot_sync(FULL_MASK, node < 0);
      const bool walked = idle == FULL_MASK && next >= count;
      bool one = false;
      if (next < count && __popc(idle) >= kLocateRefill) {
        const int i = next + __popc(idle & lt);
        if (node < 0 && i < count) {
          point = i;
          px = s_pt[w][0][i];
          py = s_pt[w][1][i];
          pz = s_pt[w][2][i];
          top = -1;
          sp = 0;
          if (A.nleaves == 1)
            one = point_in(px, py, pz, A.root_box[0], A.root_box[1], A.root_box[2], A.root_box[3], A.root_box[4],
                           A.root_box[5]);
          else
            node = 0;
        }
        next += __popc(idle);
      }
      queue(one, 0u);
#pragma unroll 1
      for (int step = 0; step < kLocateSteps; ++step) {
        bool leaf0 = false, leaf1 = false;
        int r0 = 0, r1 = 0;
        if (node >= 0) {
          const Bvh2Node *nd = A.bvh + node;
          const ChildPairs c0 = load_child<V8>(&nd->c[0]), c1 = load_child<V8>(&nd->c[1]);
          const bool h0 = point_in(px, py, pz, c0), h1 = point_in(px, py, pz, c1);
          r0 = c0.ref;
          r1 = c1.ref;
          leaf0 = h0 && r0 < 0;
          leaf1 = h1 && r1 < 0;
          const bool in0 = h0 && !leaf0, in1 = h1 && !leaf1;
          if (in0 && in1) {
            if (sp < kLocateShared) sh[sp * kLocateThreads] = top;
            else if (sp < kLocateStack) over[sp - kLocateShared] = top;
            top = r1;
            ++sp;
          }
          if (sp > kLocateStack) {
            atomicCAS(A.err, 0u, 5u);  // traversal stack overflow: the walk ends
            node = -1;
          } else if (in0 || in1) {
            node = in0 ? r0 : r1;
          } else {
            node = top;
            --sp;
            top = sp < 0 ? -1 : (sp < kLocateShared ? sh[sp * kLocateThreads] : over[sp - kLocateShared]);
          }
        }
        if (__any_sync(FULL_MASK, leaf0 || leaf1)) {
          queue(leaf0, (uint32_t)~r0);
          queue(leaf1, (uint32_t)~r1);
        }
      }
      // batches of 32; what is left once the chunk is walked, in any size
      while (true) {
        const int most = max(max(bn[0], bn[1]), max(bn[2], bn[3]));
        if (most >= 32 || (walked && qn == 0 && most > 0))
          run_bin(bn[0] == most ? 0 : (bn[1] == most ? 1 : (bn[2] == most ? 2 : 3)));
        else if (qn >= 32 || (walked && qn > 0)) classify();
        else break;
      }
      if (walked) break;
    }
    for (int i = lane; i < count; i += 32) {
      const uint32_t id = s_best[w][i];
      A.hits[base + i] = make_uint2(id, id == kNoCell ? 0u : solid_kind(A.sv.type(id)));
      if (A.rstw) A.rstw[base + i] = id == kNoCell ? make_float4(0.f, 0.f, 0.f, 0.f) : s_rst[w][i];
    }
    __syncwarp();
  }
}

}  // namespace gprtcu

using namespace gprtcu;

namespace {

bool make_view(const gprtcuSolids *s, SolidView &v) {
  if (!s) return false;
  v.n = s->numCells;
  v.vstride = s->vertexStride ? s->vertexStride : 16;
  v.istride = s->indexStride ? s->indexStride : 32;
  v.tstride = s->typeStride ? s->typeStride : 1;
  v.verts = (const unsigned char *)s->vertices;
  v.idx = (const unsigned char *)s->indices;
  v.types = (const unsigned char *)s->types;
  if (v.n == 0) return true;
  if (!v.verts || !v.idx || !v.types) return false;
  // float4 vertices (16-byte aligned, as the reference indexes them in
  // float4 units) and uint32 indices
  if (((uintptr_t)v.verts & 15) || (v.vstride & 15) || ((uintptr_t)v.idx & 3) || (v.istride & 3)) return false;
  return true;
}

}  // namespace

extern "C" GPRTCU_API gprtcuStatus gprtcuSolidBounds(const gprtcuSolids *solids, float *aabbs, float *boxes,
                                                     gprtcuStream stream) {
  SolidView v;
  if (!make_view(solids, v)) return GPRTCU_ERR_INVALID_ARG;
  if (v.n == 0) return GPRTCU_OK;
  if ((aabbs && ((uintptr_t)aabbs & 15)) || (!aabbs && !boxes)) return GPRTCU_ERR_INVALID_ARG;
  const uint64_t g = (v.n + 255) / 256, cap = (uint64_t)gprtcu_num_sms() * 16;
  k_solid_bounds<<<(unsigned)(g < cap ? g : cap), 256, 0, (cudaStream_t)stream>>>(v, (float4 *)aabbs, boxes);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuLocateSolidPoints(const gprtcuLbvh *bvh, const gprtcuSolids *solids,
                                                           const float *points, uint64_t numPoints,
                                                           gprtcuSolidHit *hits, float *rstw, void *scratch,
                                                           size_t scratchBytes, gprtcuStream stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  SolidView v;
  if (!bvh || !make_view(solids, v) || (!points && numPoints) || (!hits && numPoints)) return GPRTCU_ERR_INVALID_ARG;
  if (numPoints == 0) return GPRTCU_OK;
  if (bvh->numPrims == 0 || bvh->numPrims != v.n || !bvh->ids || !bvh->rootBox || (bvh->numPrims > 1 && !bvh->bvh2))
    return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)points & 15) || ((uintptr_t)bvh->bvh2 & 15) || ((uintptr_t)hits & 7) || ((uintptr_t)rstw & 15))
    return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  if (scratchBytes < sizeof(ScratchHeader)) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  ScratchHeader *hdr = (ScratchHeader *)scratch;
  GPRTCU_TRY(cudaMemsetAsync(scratch, 0, sizeof(ScratchHeader), stream));
  // chunks of kLocateChunk points once there are enough for every warp, else
  // an equal share, at least eight
  const uint64_t warps = (uint64_t)gprtcu_num_sms() * kLocateCtas * kLocateWarps;
  const uint64_t share = (numPoints + warps - 1) / warps;
  const int chunk = share >= kLocateChunk ? kLocateChunk : (share < 8 ? 8 : (int)share);
  const uint64_t need = (numPoints + (uint64_t)chunk * kLocateWarps - 1) / ((uint64_t)chunk * kLocateWarps);
  const int ctas = (int)(need * kLocateWarps < warps ? need : warps / kLocateWarps);
  LocateArgs a{(const Bvh2Node *)bvh->bvh2, bvh->ids, bvh->numPrims, bvh->rootBox, v, (const float4 *)points,
               numPoints, chunk, (uint2 *)hits, (float4 *)rstw,
               reinterpret_cast<unsigned long long *>(&hdr->ticket[0]), &hdr->status};
  auto launch = [&](auto kernel) { kernel<<<ctas, kLocateThreads, 0, stream>>>(a); };
  const bool v8 = ((uintptr_t)bvh->bvh2 & 31) == 0, i16 = (((uintptr_t)v.idx | v.istride) & 15) == 0;
  if (v8) i16 ? launch(k_locate_solids<true, true>) : launch(k_locate_solids<true, false>);
  else i16 ? launch(k_locate_solids<false, true>) : launch(k_locate_solids<false, false>);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}
