// wide.cu -- 8-wide BVH with 8-bit quantised child boxes, collapsed from the
// binary LBVH, and its closest-hit / any-hit traversal.  No counterpart in
// the reference (its traversal is Vulkan ray-tracing hardware); the node
// format follows the compressed-wide-BVH idea of Ylitie, Karras, Laine 2017
// ("Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
// BVHs"), written here for this library.
//
// Node (80 bytes: five 16-byte words, read in three loads, see wide_word):
//   p.xyz      fp32 origin = min corner of the children's union box
//   e.xyz      scale exponents + 127 in a byte each, scale s = 2^e per axis,
//              chosen (in FP64) as the smallest power of two with 255 * s >=
//              extent
//   imask      bit c: child slot c is an inner node
//   child_base first inner child's node index (inner children contiguous)
//   leaf_base  first leaf child's index in the wide leaf array (contiguous)
//   meta[c]    0xFF empty; else the child's rank among the inner (imask) or
//              leaf children
//   qlo/qhi    per axis, per child: floor((lo - p) / s), ceil((hi - p) / s);
//              an empty slot holds the inverted box qlo 255, qhi 0
// Traversal moves a plane's offset down (near planes) or up (far planes) with
// directed rounding and decodes it by one FMA that rounds to nearest, off by at
// most 2^-24 of its own result, which the box test's widening by 2^-18 covers:
// every decoded interval contains the exact child box's, a ray never misses a
// child that the binary traversal would enter, and intersection is the same
// FP32 watertight test, giving the same hits.  A node is 80 bytes for up to eight children
// against 64 bytes for two in the binary layout.
#include "common.cuh"
#include "lbvh.cuh"
#include "rtmath.cuh"

#include <type_traits>

uint32_t gprtcu_spin_budget(void);

namespace gprtcu {

struct __align__(16) WideNode {
  float px, py, pz;
  uint8_t ex, ey, ez;
  uint8_t imask;
  uint32_t child_base;
  uint32_t leaf_base;
  uint8_t meta[8];
  uint8_t qlo[3][8];
  uint8_t qhi[3][8];
};
static_assert(sizeof(WideNode) == 80, "80-byte wide node");

// The five 16-byte words of a node in memory: an even node has words 0..4 in
// order, an odd one word 4 first and then words 0..3, so that words (0, 1) and
// (2, 3) of every node lie on 32-byte boundaries (80-byte nodes from a 32-byte
// boundary on) and a node is three loads instead of five.  Lanes visit
// different nodes, so L1 serves a load instruction one lane per cycle
// whatever its width.
__device__ __forceinline__ uint32_t wide_word(uint32_t node, uint32_t k) {
  const uint32_t base = 5 * (node & 1u);  // position of word k within the pair of nodes
  return (node & 1u) ? (k == 4 ? base : base + 1 + k) : k;
}

struct WorkItem {
  uint32_t mesh;
  int32_t bref;  // binary inner node (mesh-local) or ~slot for a one-leaf mesh
};

// Collapse counters: the current level's items are queue[LO, HI); TAIL is
// the next free queue slot (= the number of wide nodes so far: a wide node's
// index is its queue slot), LEAF the next free wide leaf slot, TICKET the
// level kernel's CTA done-counter, EPOCH and NEXT (polled, so in a line of
// their own) the levels that the last launch has finished and TAIL after the
// latest of them, MESHES the number of roots.
enum { C_LO = 0, C_HI = 1, C_TAIL = 2, C_LEAF = 3, C_TICKET = 4, C_MESHES = 5, C_EPOCH = 32, C_NEXT = 33 };

// Levels a collapse runs: a binary node splits its keys at the highest
// differing bit of (30-bit code, 30-bit index), so binary and therefore wide
// depth stay below 62.
constexpr int kWideMaxLevels = 62;
constexpr int kWideCluster = 8;       // CTAs of the one-cluster form of the level kernel
constexpr uint32_t kWideFew = 1024;   // items that it starts a level of, with larger levels to come
constexpr uint32_t kWideMore = 4096;  // the same, once the whole-GPU levels have run

// (a box in the order of Bvh2Child::box)
__device__ __forceinline__ float box_area(const float *b) {
  const float dx = b[2] - b[0], dy = b[3] - b[1], dz = b[5] - b[4];
  return dx * dy + dy * dz + dz * dx;
}

// Smallest e with 255 * 2^e >= ext (FP64), clamped to the normal fp32 range.
__device__ __forceinline__ int frame_exponent(double ext) {
  if (!(ext > 0.0)) return -126;
  int k;
  frexp(ext / 255.0, &k);
  int e = k - 1;
  while (ldexp(255.0, e) < ext) ++e;
  while (e > -126 && ldexp(255.0, e - 1) >= ext) --e;
  return e < -126 ? -126 : (e > 127 ? 127 : e);
}

__global__ void k_wide_init(const uint32_t *tri_off, uint32_t meshes, uint32_t n, WorkItem *queue, uint32_t *roots,
                            uint32_t *counters) {
  for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < meshes; m += gridDim.x * blockDim.x) {
    const uint32_t cnt = tri_off ? tri_off[m + 1] - tri_off[m] : n;
    queue[m] = WorkItem{m, cnt == 1 ? ~0 : 0};
    roots[m] = m;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counters[C_LO] = 0;
    counters[C_HI] = meshes;
    counters[C_TAIL] = meshes;
    counters[C_LEAF] = 0;
    counters[C_TICKET] = 0;
    counters[C_MESHES] = meshes;
  }
}

// One level of the top-down collapse.  Every item of the level (a binary
// node that becomes a wide node) is expanded greedily -- the inner child of
// largest surface area is replaced by its two children until there are
// eight --, written as a quantised wide node at its queue slot, its leaf
// triangles copied to the wide leaf array and its inner children appended
// to the queue as the next level's items.  A warp allocates its children's
// queue slots and leaf slots with one atomic add each (prefix sums across
// the lanes); the last CTA to finish advances [LO, HI) to the items just
// appended.  These levels run as successive launches, so nothing waits on
// another thread's progress.  kWideClusterForm is the form for levels with few
// items (the first ones of a mesh and the last): one thread-block cluster goes
// from level to level by itself, a hardware barrier between them, while a level
// has at most `most` items.  kWideRestForm takes whatever levels are left: all
// its CTAs are on the GPU at once (a cooperative launch) and wait for one
// another after each level, `most` polls at most; a CTA whose wait runs out
// sets the call's status to GPRTCU_ERR_TIMEOUT, empties every root, since nodes
// below may not have been written, and leaves (so then do the others, and the
// last of them has emptied the roots after all that was written).  The eight candidate children stay in registers
// (unrolled loops, predicated updates) and quantising multiplies by the exact
// power of two 2^-e instead of dividing by 2^e: on 67M triangles in 16,384
// meshes the collapse went from 10.96 ms (local-memory arrays, FP64
// divisions) to 5.43 ms with the same nodes.  The candidates' boxes then
// moved to thread-private shared memory (72 instead of 125 registers, 7 CTAs
// per SM instead of 4): 4.8 ms.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
enum { kWideLevelForm, kWideClusterForm, kWideRestForm };
template <int FORM>
__global__ void __launch_bounds__(128, FORM == kWideClusterForm ? 1 : 7) k_wide_level(const Bvh2Node *bvh2, const float4 *leaf_tris,
                                                    const uint32_t *tri_off, WideNode *wnodes, float4 *wleaf,
                                                    WorkItem *queue, uint32_t *counters, uint32_t most) {
  uint32_t lo = counters[C_LO], hi = counters[C_HI];
  // an empty level appends nothing, so the next window equals this one: the
  // launch leaves the counters as they are
  if (lo == hi || (FORM == kWideClusterForm && hi - lo > most)) return;
  const int lane = threadIdx.x & 31;
  // candidate child boxes, thread-private: [coordinate][slot][thread]
  __shared__ float s_box[6][8][128];
#define CBOX(c, k) s_box[(k)][(c)][threadIdx.x]
  const uint32_t stride = gridDim.x * blockDim.x;
  for (int level = 0; level < (FORM == kWideLevelForm ? 1 : kWideMaxLevels); ++level) {
    const uint32_t total = hi - lo;
    for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < total; i0 += stride) {
      const uint32_t idx = lo + i0 + lane;
      const bool valid = i0 + lane < total;
      // References and areas live in registers (every index below is a
      // compile-time slot number: unrolled loops with predicated updates), the
      // boxes in this thread's column of s_box, so nothing goes to local memory.
      int ref[8];
      float area[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        ref[c] = -1;
        area[c] = 0.0f;
      }
      int cnt = 0;
      uint32_t m = 0, b = 0;
      if (valid) {
        const WorkItem it = queue[idx];
        m = it.mesh;
        b = tri_off ? tri_off[m] : 0u;
        const Bvh2Node *mb = bvh2 + (b - m);
        if (it.bref < 0) {
          const uint32_t slot = (uint32_t)~it.bref;
          const float4 a = leaf_tris[3 * (size_t)(b + slot)], c = leaf_tris[3 * (size_t)(b + slot) + 1],
                       d = leaf_tris[3 * (size_t)(b + slot) + 2];
          ref[0] = it.bref;
          CBOX(0, 0) = fminf(a.x, fminf(c.x, d.x));
          CBOX(0, 1) = fminf(a.y, fminf(c.y, d.y));
          CBOX(0, 2) = fminf(a.z, fminf(c.z, d.z));
          CBOX(0, 3) = fmaxf(a.x, fmaxf(c.x, d.x));
          CBOX(0, 4) = fmaxf(a.y, fmaxf(c.y, d.y));
          CBOX(0, 5) = fmaxf(a.z, fmaxf(c.z, d.z));
          cnt = 1;
        } else {
          const Bvh2Node nd = mb[it.bref];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            ref[c] = nd.c[c].ref;
#pragma unroll
            for (int k = 0; k < 6; ++k) CBOX(c, k) = nd.c[c].box[box_word(k)];
            area[c] = box_area(nd.c[c].box);
          }
          cnt = 2;
          // greedy: replace the inner child of largest area (lowest slot on
          // ties) by its two children until there are eight
          while (cnt < 8) {
            int best = -1;
            float ba = -1.0f;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (c < cnt && ref[c] >= 0 && area[c] > ba) {
                ba = area[c];
                best = c;
              }
            if (best < 0) break;
            int rb = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (c == best) rb = ref[c];
            const Bvh2Node ch = mb[rb];
            const float a0 = box_area(ch.c[0].box), a1 = box_area(ch.c[1].box);
#pragma unroll
            for (int k = 0; k < 6; ++k) {
              CBOX(best, k) = ch.c[0].box[box_word(k)];
              CBOX(cnt, k) = ch.c[1].box[box_word(k)];
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              if (c == best) {
                ref[c] = ch.c[0].ref;
                area[c] = a0;
              }
              if (c == cnt) {
                ref[c] = ch.c[1].ref;
                area[c] = a1;
              }
            }
            ++cnt;
          }
        }
      }
      uint32_t n_inner = 0, n_leaf = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < cnt) (ref[c] >= 0 ? n_inner : n_leaf)++;
      // warp-aggregated allocation of child queue slots and leaf slots
      const uint32_t inc_i = warp_incl_scan(n_inner, lane), inc_l = warp_incl_scan(n_leaf, lane);
      const uint32_t tot_i = __shfl_sync(FULL_MASK, inc_i, 31), tot_l = __shfl_sync(FULL_MASK, inc_l, 31);
      uint32_t base_i = 0, base_l = 0;
      if (lane == 0) {
        if (tot_i) base_i = atomicAdd(&counters[C_TAIL], tot_i);
        if (tot_l) base_l = atomicAdd(&counters[C_LEAF], tot_l);
      }
      base_i = __shfl_sync(FULL_MASK, base_i, 0);
      base_l = __shfl_sync(FULL_MASK, base_l, 0);
      if (!valid) continue;
      const uint32_t child_base = base_i + inc_i - n_inner, leaf_base = base_l + inc_l - n_leaf;
      float lo3[3] = {CBOX(0, 0), CBOX(0, 1), CBOX(0, 2)}, hi3[3] = {CBOX(0, 3), CBOX(0, 4), CBOX(0, 5)};
#pragma unroll
      for (int c = 1; c < 8; ++c)
        if (c < cnt)
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            lo3[k] = fminf(lo3[k], CBOX(c, k));
            hi3[k] = fmaxf(hi3[k], CBOX(c, 3 + k));
          }
      int e[3];
      double isc[3];  // 2^-e: dividing by the scale 2^e is this exact product
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        e[k] = frame_exponent((double)hi3[k] - (double)lo3[k]);
        isc[k] = ldexp(1.0, -e[k]);
      }
      uint32_t imask = 0, meta_w[2] = {0u, 0u}, qlo_w[3][2] = {{0u, 0u}, {0u, 0u}, {0u, 0u}},
               qhi_w[3][2] = {{0u, 0u}, {0u, 0u}, {0u, 0u}};
      uint32_t ri = 0, rl = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int h = c >> 2, sh = 8 * (c & 3);
        // an absent child is the inverted box (lo 255, hi 0): it fails the slab test
        uint32_t meta = 0xFF, ql[3] = {255u, 255u, 255u}, qh[3] = {0u, 0u, 0u};
        if (c < cnt) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const double l = floor(((double)CBOX(c, k) - (double)lo3[k]) * isc[k]);
            const double u = ceil(((double)CBOX(c, 3 + k) - (double)lo3[k]) * isc[k]);
            ql[k] = (uint32_t)(l < 0.0 ? 0.0 : (l > 255.0 ? 255.0 : l));
            qh[k] = (uint32_t)(u < 0.0 ? 0.0 : (u > 255.0 ? 255.0 : u));
          }
          if (ref[c] >= 0) {
            imask |= 1u << c;
            meta = ri;
            queue[child_base + ri] = WorkItem{m, ref[c]};  // the next level's item; its wide node index
            ++ri;
          } else {
            const uint32_t slot = (uint32_t)~ref[c];
            const size_t src = 3 * (size_t)(b + slot), dst = 3 * (size_t)(leaf_base + rl);
            wleaf[dst] = leaf_tris[src];
            wleaf[dst + 1] = leaf_tris[src + 1];
            wleaf[dst + 2] = leaf_tris[src + 2];
            meta = rl;
            ++rl;
          }
        }
        meta_w[h] |= meta << sh;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          qlo_w[k][h] |= ql[k] << sh;
          qhi_w[k][h] |= qh[k] << sh;
        }
      }
      // the 80-byte node as five 16-byte words (layout of WideNode, wide_word)
      uint4 *op = reinterpret_cast<uint4 *>(wnodes) + 5 * (size_t)(idx & ~1u);
      op[wide_word(idx, 0)] = make_uint4(__float_as_uint(lo3[0]), __float_as_uint(lo3[1]), __float_as_uint(lo3[2]),
                                         (uint32_t)(e[0] + 127) | ((uint32_t)(e[1] + 127) << 8) |
                                             ((uint32_t)(e[2] + 127) << 16) | (imask << 24));
      op[wide_word(idx, 1)] = make_uint4(child_base, leaf_base, meta_w[0], meta_w[1]);
      op[wide_word(idx, 2)] = make_uint4(qlo_w[0][0], qlo_w[0][1], qlo_w[1][0], qlo_w[1][1]);
      op[wide_word(idx, 3)] = make_uint4(qlo_w[2][0], qlo_w[2][1], qhi_w[0][0], qhi_w[0][1]);
      op[wide_word(idx, 4)] = make_uint4(qhi_w[1][0], qhi_w[1][1], qhi_w[2][0], qhi_w[2][1]);
    }
    if constexpr (FORM == kWideRestForm) {
      // the last CTA to finish the level tells the others how many items the
      // next one has
      __shared__ uint32_t s_next;
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        uint32_t next = 0;
        if (atomicAdd(&counters[C_TICKET], 1u) == gridDim.x - 1) {
          __threadfence();
          next = ld_relaxed_u32(&counters[C_TAIL]);
          st_relaxed_u32(&counters[C_TICKET], 0u);
          st_relaxed_u32(&counters[C_NEXT], next);
          __threadfence();
          st_relaxed_u32(&counters[C_EPOCH], (uint32_t)level + 1u);
        } else {
          bool ok = false;
          for (uint32_t i = 0; !ok && i <= most; ++i) ok = ld_acquire_u32(&counters[C_EPOCH]) > (uint32_t)level;
          if (ok) next = ld_relaxed_u32(&counters[C_NEXT]);
          else record_error(reinterpret_cast<ScratchHeader *>(reinterpret_cast<char *>(counters) - sizeof(ScratchHeader)),
                            GPRTCU_ERR_TIMEOUT);
        }
        s_next = next;
      }
      __syncthreads();
      const uint32_t tail = s_next;
      if (tail == 0)  // the wait ran out
        for (uint32_t m = threadIdx.x; m < counters[C_MESHES]; m += blockDim.x) {
          uint4 *op = reinterpret_cast<uint4 *>(wnodes) + 5 * (size_t)(m & ~1u);
          op[wide_word(m, 0)] = make_uint4(0u, 0u, 0u, 0u);
          op[wide_word(m, 1)] = make_uint4(0u, 0u, ~0u, ~0u);
          op[wide_word(m, 2)] = make_uint4(~0u, ~0u, ~0u, ~0u);
          op[wide_word(m, 3)] = make_uint4(~0u, ~0u, 0u, 0u);
          op[wide_word(m, 4)] = make_uint4(0u, 0u, 0u, 0u);
        }
      if (tail <= hi) break;  // no items left
      lo = hi;
      hi = tail;
    }
    if constexpr (FORM == kWideClusterForm) {
      cluster_sync();  // the next level's items are written
      const uint32_t tail = ld_relaxed_u32(&counters[C_TAIL]);
      cluster_sync();  // and everyone knows how many before they append to them
      lo = hi;
      hi = tail;
      if (lo == hi || hi - lo > most) break;
    }
  }
#undef CBOX
  if constexpr (FORM == kWideClusterForm) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      counters[C_LO] = lo;
      counters[C_HI] = hi;
    }
  }
  if constexpr (FORM != kWideLevelForm) return;
  // the last CTA to finish moves the level window to the appended items
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&counters[C_TICKET], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    counters[C_LO] = hi;
    counters[C_HI] = ld_relaxed_u32(&counters[C_TAIL]);
    counters[C_TICKET] = 0;
  }
}

// ---------------------------------------------------------------------------
// traversal
// ---------------------------------------------------------------------------
constexpr int kWideThreads = 128;
constexpr int kWideStack = 64;
constexpr int kWideCtas = 7;    // per SM: 72 registers
constexpr int kWideShared = 6;  // stack entries in shared memory
constexpr int kWideRefill = 6;

// 2^16 x the quantisation step of axis 0..2 from a node's word of biased
// exponents (infinity past the float range: the axis then gives NaN and drops
// out of the box test, which stays conservative).
template <int AXIS> __device__ __forceinline__ float scale16_of(uint32_t w) {
  return __fmul_rn(__uint_as_float((AXIS == 0 ? w << 23 : (AXIS == 1 ? w << 15 : w << 7)) & 0x7F800000u), 65536.0f);
}

// Largest m < meshes with off[m] <= r, given off[m0] <= r: gallop upward
// from m0, then bisect.  off has meshes + 1 entries, off[meshes] > r.
__device__ __forceinline__ uint32_t mesh_from(const uint32_t *off, uint32_t meshes, uint32_t m0, uint64_t r) {
  uint32_t lo = m0, hi = m0 + 1, step = 1;
  while (hi < meshes && __ldg(off + hi) <= r) {
    lo = hi;
    step <<= 1;
    hi = lo + step;
  }
  if (hi > meshes) hi = meshes;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(off + mid) <= r) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Lane refill.  When at least kWideRefill lanes of a warp are idle (or all
// are), the warp takes that many new rays from the global counter (waiting
// for the whole warp to finish left most lanes idle behind the longest ray).
// On 16.7M rays of one 16.7M-triangle mesh and on 134M rays over 16,384
// meshes, thresholds of 4, 8, 16 and 32 (no refill) idle lanes measured
// 33.6 / 34.7 / 38.5 / 63.7 ms and 71.3 / 69.0 / 74.8 / 155.5 ms.  The
// counter only grows, so the mesh of the first new ray is at or after the
// warp's previous mesh: the 32 lanes probe the next 32 mesh offsets at once
// (one load latency instead of a serial gallop), and a lane whose ray lies
// before the end of that mesh needs no search of its own.  Called by all 32
// lanes; returns true on the lanes that took a ray (their traversal state is
// then reset by the caller).
template <bool BATCHED>
__device__ __forceinline__ bool wide_take_ray(bool &active, bool &drained, uint32_t &warp_mesh, uint64_t &r,
                                              Ray &R, uint32_t &node, const uint32_t *roots,
                                              const uint32_t *ray_off, uint32_t meshes, const float4 *rays,
                                              uint64_t nrays, unsigned long long *counter) {
  const int lane = threadIdx.x & 31;
  const unsigned idle = __ballot_sync(FULL_MASK, !active);
  const int n_idle = __popc(idle);
  if (drained || (n_idle < kWideRefill && n_idle != 32)) return false;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(counter, (unsigned long long)n_idle);
  base = __shfl_sync(FULL_MASK, base, 0);
  if (base + n_idle >= nrays) drained = true;
  uint64_t mesh_end = 0;  // first ray after warp_mesh
  if (BATCHED && base < nrays) {
    while (true) {
      const uint32_t j = warp_mesh + 1 + lane;
      const uint32_t v = j <= meshes ? __ldg(ray_off + j) : 0xFFFFFFFFu;
      const int k = __popc(__ballot_sync(FULL_MASK, j < meshes && v <= base));  // a prefix of the lanes
      warp_mesh += k;
      if (k < 32) {
        mesh_end = __shfl_sync(FULL_MASK, v, k);
        break;
      }
    }
  }
  if (active) return false;
  const uint64_t mine = base + __popc(idle & ((1u << lane) - 1u));
  if (mine >= nrays) return false;
  r = mine;
  active = true;
  ray_setup(__ldg(rays + 2 * r), __ldg(rays + 2 * r + 1), R);
  uint32_t m = 0;
  if (BATCHED) m = mine < mesh_end ? warp_mesh : mesh_from(ray_off, meshes, warp_mesh, r);
  node = __ldg(roots + m);
  return true;
}

// One node step: the ray is moved into the node's quantised frame once, the
// eight child boxes are tested two at a time with packed f32x2 arithmetic
// (byte decode, slab FMAs, the 2^-18 widening) and three-input min/max (68.7
// -> 60.7 ms on 134 M rays over 16,384 meshes against the scalar loop).  A
// plane byte q is decoded by one instruction into the float v = 1 + q 2^-16;
// with M = 2^16 x the step in t and the plane offset moved down (near planes)
// or up (far planes) by M in that direction of rounding, one FMA v M + (offset
// - M) gives q x step + offset without a separate bias subtraction (47.8 ->
// 47.2 ms).  The FMA rounds once, to nearest: it is off by 2^-24 of its own
// result, which the widening by 2^-18 covers (only the offset's error is not
// relative to the result, hence its directed steps); packed FMAs with directed
// rounding cost two scalar ones each.  Absent children are inverted boxes and
// need no test of their own.  What bounds the step is the ALU pipe (75 % busy:
// byte permutes, min/max, selects), so the bytes are decoded on the FMA pipe
// (wide_plane: 4.29 -> 4.02 ms on 4.0 M rays of 4.2 M triangles, 24.9 -> 24.2
// ms on 77.5 M rays over 4,096 meshes), a child's test puts the sign of exit - entry
// into the miss mask by one funnel shift instead of a compare and a predicated
// OR, and the nearest hit inner child (NEAREST: entering the lowest hit slot
// instead measured 40.3 against 22.7 ms on 16.8 M rays of one 16.8
// M-triangle mesh) is one predicated integer min per child over the entry
// distance's bits with the slot in the lowest three: 4.60 -> 4.33 ms on 4.0 M
// rays of 4.2 M triangles.  Without NEAREST the lowest hit inner slot is
// entered (any hit: 16.8 against 17.7 ms on the same rays).  An exit that
// underflows to -0 counts as behind the ray.
struct WideStep {
  uint32_t hm;  // slots whose box is hit
  uint32_t imask, child_base, leaf_base, meta_lo, meta_hi;
  int ns;  // nearest hit inner slot, -1 if none
};

// Words 2k and 2k + 1 of a node's first four (p on a 32-byte boundary when V8).
template <bool V8> __device__ __forceinline__ void load_words(const uint4 *p, uint4 &a, uint4 &b) {
  if constexpr (V8) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
        : "l"(p));
  } else {
    a = __ldg(p);
    b = __ldg(p + 1);
  }
}

// Plane byte c of a word as the float 1 + q 2^-16: the dot product with one
// byte 128 added to the bits of 1.0.  It runs on the FMA pipe, where a byte
// permute is one of the ALU pipe's 250 instructions per step.
__device__ __forceinline__ float wide_plane(uint32_t q, int c) {
  return __uint_as_float(__dp4a(q, 128u << (8 * (c & 3)), 0x3F800000u));
}

template <bool NEAREST, bool V8>
__device__ __forceinline__ WideStep wide_node_step(const WideNode *nodes, uint32_t node, const Ray &R, float bt) {
  WideStep S;
  const uint4 *np = reinterpret_cast<const uint4 *>(nodes + node);
  const uint32_t odd = node & 1u;
  uint4 w0, w1, w2, w3;
  load_words<V8>(np + odd, w0, w1);
  load_words<V8>(np + odd + 2, w2, w3);
  const uint4 w4 = __ldg(np + (odd ? 0 : 4));
  const float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
  const float sx = scale16_of<0>(w0.w), sy = scale16_of<1>(w0.w), sz = scale16_of<2>(w0.w);
  S.imask = w0.w >> 24;
  S.child_base = w1.x;
  S.leaf_base = w1.y;
  S.meta_lo = w1.z;
  S.meta_hi = w1.w;
  float An[3], Af[3], Bq[3];
  uint32_t qn[3][2], qf[3][2];
  {
    const float pa[3] = {px, py, pz}, oa[3] = {R.ox, R.oy, R.oz}, ia[3] = {R.ix, R.iy, R.iz};
    const float sa[3] = {sx, sy, sz};
    const uint32_t ql[3][2] = {{w2.x, w2.y}, {w2.z, w2.w}, {w3.x, w3.y}};
    const uint32_t qh[3][2] = {{w3.z, w3.w}, {w4.x, w4.y}, {w4.z, w4.w}};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float dlo = __fsub_rd(pa[a], oa[a]), dhi = __fsub_ru(pa[a], oa[a]);
      const bool pos = !(ia[a] < 0.0f);
      An[a] = __fmul_rd(pos ? dlo : dhi, ia[a]);
      Af[a] = __fmul_ru(pos ? dhi : dlo, ia[a]);
      Bq[a] = __fmul_rn(sa[a], ia[a]);  // M: 2^16 x the step in t (exactly 2^16 x the rounded step)
      An[a] = __fsub_rd(An[a], Bq[a]);
      Af[a] = __fsub_ru(Af[a], Bq[a]);
      qn[a][0] = pos ? ql[a][0] : qh[a][0];
      qn[a][1] = pos ? ql[a][1] : qh[a][1];
      qf[a][0] = pos ? qh[a][0] : ql[a][0];
      qf[a][1] = pos ? qh[a][1] : ql[a][1];
    }
  }
  // The children from the last to the first: a miss puts the sign of (exit -
  // entry) into the miss mask by one funnel shift.
  uint32_t miss = 0;
  float tn[8];
  {
    const unsigned long long lo2 = pk2(kBoxLo, kBoxLo), hi2 = pk2(kBoxHi, kBoxHi), neg2 = pk2(-1.0f, -1.0f);
    unsigned long long B2[3], N2[3], F2[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      B2[a] = pk2(Bq[a], Bq[a]);
      N2[a] = pk2(An[a], An[a]);
      F2[a] = pk2(Af[a], Af[a]);
    }
#pragma unroll
    for (int cp = 3; cp >= 0; --cp) {
      const int h = cp >> 1;
      float n[2][3], f[2][3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const unsigned long long qn2 = pk2(wide_plane(qn[a][h], 2 * cp), wide_plane(qn[a][h], 2 * cp + 1));
        const unsigned long long qf2 = pk2(wide_plane(qf[a][h], 2 * cp), wide_plane(qf[a][h], 2 * cp + 1));
        up2(fma2_rn(qn2, B2[a], N2[a]), n[0][a], n[1][a]);
        up2(fma2_rn(qf2, B2[a], F2[a]), f[0][a], f[1][a]);
      }
      float tf[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        tn[2 * cp + k] = fmaxf(max3f(n[k][0], n[k][1], n[k][2]), R.tmin);
        tf[k] = min3f(f[k][0], f[k][1], f[k][2]);
      }
      const unsigned long long e2 = mul2_rn(pk2(tn[2 * cp], tn[2 * cp + 1]), lo2);
      up2(e2, tn[2 * cp], tn[2 * cp + 1]);
      up2(mul2_rn(pk2(tf[0], tf[1]), hi2), tf[0], tf[1]);
      // the widened exit clamped by the best distance: one test per child
      tf[0] = fminf(tf[0], bt);
      tf[1] = fminf(tf[1], bt);
      float d[2];
      up2(fma2_rn(e2, neg2, pk2(tf[0], tf[1])), d[0], d[1]);
      miss = __funnelshift_l(__float_as_uint(d[1]), miss, 1);
      miss = __funnelshift_l(__float_as_uint(d[0]), miss, 1);
    }
  }
  const uint32_t hm = ~miss & 0xFFu;
  S.hm = hm;
  const uint32_t inner = hm & S.imask;
  if constexpr (NEAREST) {
    // nearest hit inner child: entry distances (not negative, so their bits
    // order as integers do) with the slot in the three lowest bits
    uint32_t best = 0xFFFFFFFFu;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (inner & (1u << c)) best = min(best, (__float_as_uint(tn[c]) & ~7u) | (uint32_t)c);
    S.ns = inner ? (int)(best & 7u) : -1;
  } else {
    S.ns = inner ? __ffs(inner) - 1 : -1;
  }
  return S;
}

// The next node: the nearest hit inner child is entered and the other hit
// inner children are pushed as one entry {child_base, slot mask | inner mask
// << 8} (a popped slot's node is child_base + the inner children below it);
// with no inner child hit, the top entry's lowest slot is popped.  The top
// entry stays in registers (slot mask zero: none), the next SHARED below it in
// shared memory, the rest in local memory.  Returns false when the traversal
// is over (or the stack overflowed: status 5).
template <int SHARED>
__device__ __forceinline__ bool wide_next(const WideStep &S, uint2 &top, uint2 *sh, uint2 *over, int &sp,
                                          uint32_t &node, uint32_t *err) {
  if (S.ns >= 0) {
    const uint32_t rest = S.hm & S.imask & ~(1u << S.ns);
    if (rest) {
      if (top.y & 0xFFu) {
        if (sp < SHARED) sh[sp * kWideThreads] = top;
        else if (sp < kWideStack) over[sp - SHARED] = top;
        else {
          atomicCAS(err, 0u, 5u);  // traversal stack overflow
          return false;
        }
        ++sp;
      }
      top = make_uint2(S.child_base, rest | (S.imask << 8));
    }
    node = S.child_base + (uint32_t)__popc(S.imask & ((1u << S.ns) - 1u));
    return true;
  }
  if (!(top.y & 0xFFu)) return false;
  const uint32_t c = __ffs(top.y & 0xFFu) - 1;
  node = top.x + (uint32_t)__popc((top.y >> 8) & ((1u << c) - 1u));
  top.y &= ~(1u << c);
  if (!(top.y & 0xFFu) && sp > 0) {
    --sp;
    top = sp < SHARED ? sh[sp * kWideThreads] : over[sp - SHARED];
  }
  return true;
}

// The top bits of a word's four bytes, in order.
__device__ __forceinline__ uint32_t wide_msbs(uint32_t w) { return (((w >> 7) & 0x01010101u) * 0x01020408u) >> 24; }

// A finished ray's record: the primitive id and, until k_wide_refine
// replaces it by t, the leaf slot of the triangle hit.
__device__ __forceinline__ Hit wide_result(uint32_t best, uint32_t best_leaf) {
  Hit out;
  out.prim = best;
  out.t = best != kMiss ? __uint_as_float(best_leaf) : __int_as_float(0x7f800000);
  return out;
}

// t of every hit: the plane-equation distance of the hit triangle in
// double-float, rounded once.  Run after the traversal over all rays at once
// instead of by each lane as its ray finished (when few lanes of the warp ran
// it and the rest waited).  A warp reads 32 records at a time (coalesced)
// and queues the indices of the hits in shared memory; every 32 queued hits
// are refined with all lanes busy (a lane per record left ~1 in 5 busy: 2.0
// ms cold for 134M rays, 18 % of them hits).
constexpr int kRefineThreads = 256;

__global__ void __launch_bounds__(kRefineThreads) k_wide_refine(const float4 *leaf, const float4 *rays,
                                                                uint64_t nrays, Hit *hits) {
  __shared__ uint64_t s_q[kRefineThreads / 32][64];
  const int lane = threadIdx.x & 31;
  uint64_t *q = s_q[threadIdx.x >> 5];
  auto refine = [&](int count) {
    __syncwarp();
    if (lane < count) {
      const uint64_t i = q[lane];
      const uint32_t slot = __float_as_uint(hits[i].t);
      const float4 o = __ldg(rays + 2 * i), d = __ldg(rays + 2 * i + 1);
      Ray R;
      R.ox = o.x;
      R.oy = o.y;
      R.oz = o.z;
      R.dx = d.x;
      R.dy = d.y;
      R.dz = d.z;
      const float4 a = __ldg(leaf + 3 * (size_t)slot), b = __ldg(leaf + 3 * (size_t)slot + 1),
                   c = __ldg(leaf + 3 * (size_t)slot + 2);
      const float v0[3] = {a.x, a.y, a.z}, v1[3] = {b.x, b.y, b.z}, v2[3] = {c.x, c.y, c.z};
      hits[i].t = refine_t(R, v0, v1, v2);
    }
    __syncwarp();
  };
  int nq = 0;  // queued hits, the same on every lane
  const uint64_t warps = (uint64_t)gridDim.x * (kRefineThreads / 32);
  for (uint64_t base = (blockIdx.x * (uint64_t)(kRefineThreads / 32) + (threadIdx.x >> 5)) * 32; base < nrays;
       base += warps * 32) {
    const uint64_t i = base + lane;
    const bool hit = i < nrays && hits[i].prim != kMiss;
    const unsigned m = __ballot_sync(FULL_MASK, hit);
    if (hit) q[nq + __popc(m & ((1u << lane) - 1u))] = i;
    nq += __popc(m);
    if (nq >= 32) {
      refine(32);
      const uint64_t v = lane < nq - 32 ? q[32 + lane] : 0;
      __syncwarp();
      if (lane < nq - 32) q[lane] = v;
      nq -= 32;
    }
  }
  refine(nq);
}

constexpr int kWideFlush = 16;  // queued entries that trigger a flush
constexpr int kWideSteps = 3;   // node steps between two looks at what else is to be done
constexpr int kWideQueue = kWideFlush + 32 * kWideSteps;  // a step queues at most 32 entries

// Closest hit: one lane per ray, and the triangle tests of the hit leaf
// children are queued per warp in shared memory instead of being run at once
// (a node step hits about one leaf triangle per 14 lanes, so running the tests
// at once kept ~2 of 32 lanes busy for the length of a triangle test in most
// steps).  A step's hit leaves are one entry, {leaf_base, hit slots | inner
// mask << 8 | lane << 16}.  When kWideFlush entries are queued their tests are
// listed and run by all 32 lanes (the owner's ray comes by shuffles and from
// shared memory), each hit folded into the owner's best (t, id) key with one
// shared-memory atomicMin; the owners then take the key's t as their culling
// distance.  A lane whose traversal is over while tests of its ray are still
// queued waits for the flush, which also runs when no lane of the warp
// traverses any more, or when the waiting lanes and the idle ones add up to a
// refill.  The closest (t, id) over all tested triangles is the same in any
// order of tests, so the hits equal the immediate test's; the culling
// distance only lags.
// Any hit (ANY) walks on while its tests are queued, and the first entry of a
// ray with a hit ends it: the key's upper word is then the entry's place in
// the queue, so the hit is the one that tests run at once would have found
// (the closest of that entry, ties to the lowest id).  Tests run at once
// left 16.6 of 32 lanes active: 4.0 M rays on 4.2 M triangles 3.82 -> 3.08 ms
// with the changes to the step above, 77.5 M rays over 4,096 meshes 25.0 ->
// 20.3 ms.
// One entry per lane and step (placing every test by a prefix sum over the
// lanes in every step took as long as the tests), kWideSteps steps between two
// looks at flush, refill and finished rays, and 72 registers without spills:
// 4.0 M rays on 4.2 M triangles 5.08 -> 4.30 ms with the changes to the step
// above, 77.5 M rays over 4,096 meshes 28.6 -> 24.9 ms, 1,048,576 rays on
// 262,144 triangles 1.58 -> 1.33 ms.  7 / 8 / 9 CTAs per SM (72 / 64 / 56
// registers, the last spilling): 4.33 / 4.44 / 4.61 ms; 1 / 2 / 3 / 4 / 5 / 8
// steps: 4.83 / 4.45 / 4.44 / 4.39 / 4.59 / 4.66 ms; flush at 10 / 16 / 24
// entries: 4.63 / 4.60 / 4.69 ms; refill at 4 / 6 / 8 idle lanes: 4.30 / 4.30
// / 4.37 ms, and 25.2 / 24.9 / 24.8 ms on the 4,096 meshes.
template <bool ANY, bool BATCHED, bool V8>
__global__ void __launch_bounds__(kWideThreads, kWideCtas)
    k_trace_wide(const WideNode *nodes, const float4 *leaf, const uint32_t *roots, const uint32_t *ray_off,
                         uint32_t meshes, const float4 *rays, uint64_t nrays, Hit *hits,
                         unsigned long long *counter, uint32_t *err) {
  __shared__ uint2 s_stack[kWideShared][kWideThreads];
  __shared__ uint2 s_queue[kWideThreads / 32][kWideQueue];
  __shared__ uint8_t s_list[kWideThreads / 32][256];  // tests of 32 entries: entry | slot << 5
  __shared__ unsigned long long s_best[kWideThreads / 32][32];
  __shared__ uint32_t s_bslot[kWideThreads / 32][32];
  __shared__ uint32_t s_bid[kWideThreads / 32][ANY ? 32 : 1];  // any hit: the primitive of s_best
  // what only the flush and the final store read stays in shared memory, not
  // in registers
  __shared__ float s_rs[kWideThreads / 32][4][32];  // Sx, Sy, Sz, tmax of each lane's ray
  __shared__ int s_rk[kWideThreads / 32][32];        // kx | ky << 2 | kz << 4
  __shared__ unsigned long long s_rid[kWideThreads / 32][32];  // ray index
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint2 *queue = s_queue[wq];
  uint8_t *list = s_list[wq];
  unsigned long long *sbest = s_best[wq];
  uint32_t *sbslot = s_bslot[wq];
  bool active = false, drained = false, walking = false, pending = false;
  uint64_t r = 0;
  Ray R;
  uint32_t node = 0;
  float bt = 0.0f;
  uint2 *const sh = &s_stack[0][threadIdx.x];
  uint2 over[kWideStack - kWideShared], top = make_uint2(0u, 0u);
  uint32_t warp_mesh = 0;
  int sp = 0, nq = 0;  // nq: queued entries, the same on every lane

  // Runs the queued tests with all lanes (warp-uniform call).
  auto flush = [&]() {
    __syncwarp();
    for (int b = 0; b < nq; b += 32) {
      const uint2 v = b + lane < nq ? queue[b + lane] : make_uint2(0u, 0u);
      uint32_t bits = v.y & 0xFFu;
      const uint32_t cnt = __popc(bits), inc = warp_incl_scan(cnt, lane);
      const int total = (int)__shfl_sync(FULL_MASK, inc, 31);
      for (uint32_t k = inc - cnt; bits; bits &= bits - 1u) list[k++] = (uint8_t)(lane | ((__ffs(bits) - 1) << 5));
      __syncwarp();
      for (int k = 0; k < total; k += 32) {
        const bool on = k + lane < total;
        const uint32_t code = on ? list[k + lane] : (uint32_t)lane;
        const uint32_t ex = __shfl_sync(FULL_MASK, v.x, code & 31u), ey = __shfl_sync(FULL_MASK, v.y, code & 31u);
        const int o = on ? (int)(ey >> 16) : lane;
        // a leaf's rank among the node's leaves: the slots below it that are
        // not inner (empty slots come last)
        const uint32_t slot = ex + (uint32_t)__popc(~(ey >> 8) & ((1u << (code >> 5)) - 1u));
        Ray Q;
        Q.ox = __shfl_sync(FULL_MASK, R.ox, o);
        Q.oy = __shfl_sync(FULL_MASK, R.oy, o);
        Q.oz = __shfl_sync(FULL_MASK, R.oz, o);
        Q.tmin = __shfl_sync(FULL_MASK, R.tmin, o);
        Q.Sx = s_rs[wq][0][o];
        Q.Sy = s_rs[wq][1][o];
        Q.Sz = s_rs[wq][2][o];
        Q.tmax = s_rs[wq][3][o];
        const int kk = s_rk[wq][o];
        Q.kx = kk & 3;
        Q.ky = (kk >> 2) & 3;
        Q.kz = kk >> 4;
        unsigned long long key = ~0ull;
        uint32_t id = 0;
        if (on) {
          const float4 a = __ldg(leaf + 3 * (size_t)slot), bb = __ldg(leaf + 3 * (size_t)slot + 1),
                       c = __ldg(leaf + 3 * (size_t)slot + 2);
          const float v0[3] = {a.x, a.y, a.z}, v1[3] = {bb.x, bb.y, bb.z}, v2[3] = {c.x, c.y, c.z};
          float t;
          id = __float_as_uint(a.w);
          if (isect_tri(Q, v0, v1, v2, t)) {
            key = ANY ? ((unsigned long long)(b + (int)(code & 31u)) << 32) | t_order(t)
                      : ((unsigned long long)t_order(t) << 32) | id;
            if (!ANY) atomicMin(&sbest[o], key);
          }
        }
        unsigned long long before = 0;  // any hit: the key that s_bid belongs to
        if constexpr (ANY) {
          before = sbest[o];
          __syncwarp();
          if (key != ~0ull) atomicMin(&sbest[o], key);
        }
        __syncwarp();
        bool won = key != ~0ull && sbest[o] == key;
        if constexpr (ANY) {
          // the same entry and distance: the lowest id, over all 32-test
          // batches that the entry's tests are in
          if (won && before != key) s_bid[wq][o] = kMiss;
          __syncwarp();
          if (won) atomicMin(&s_bid[wq][o], id);
          __syncwarp();
          won = won && s_bid[wq][o] == id;
        }
        if (won) sbslot[o] = slot;  // one winner per owner
        __syncwarp();
      }
    }
    if (pending) {
      if (!ANY) bt = t_from_order((uint32_t)(sbest[lane] >> 32));
      else if (sbest[lane] != ~0ull) walking = false;
      pending = false;
    }
    nq = 0;
  };

  while (true) {
    if (wide_take_ray<BATCHED>(active, drained, warp_mesh, r, R, node, roots, ray_off, meshes, rays, nrays,
                               counter)) {
      bt = __fadd_rn(R.tmax, 0.0f);  // never -0 (wide_node_step tests a sign)
      sp = 0;
      top.y = 0;
      walking = true;
      sbest[lane] = ANY ? ~0ull : ((unsigned long long)t_order(R.tmax) << 32) | kMiss;
      s_rs[wq][0][lane] = R.Sx;
      s_rs[wq][1][lane] = R.Sy;
      s_rs[wq][2][lane] = R.Sz;
      s_rs[wq][3][lane] = R.tmax;
      s_rk[wq][lane] = R.kx | (R.ky << 2) | (R.kz << 4);
      s_rid[wq][lane] = r;
    }
    if (!__any_sync(FULL_MASK, active)) {
      if (drained) break;
      continue;
    }
#pragma unroll 1
    for (int step = 0; step < kWideSteps; ++step) {
      uint32_t lh = 0, lbase = 0;
      if (walking) {
        const WideStep S = wide_node_step<!ANY, V8>(nodes, node, R, bt);
        lbase = S.leaf_base;
        lh = S.hm & ~S.imask;
        // an empty slot (meta 0xFF; only an infinite scale lets one pass the
        // box test) is no leaf
        if (lh) lh = (lh & ~(wide_msbs(S.meta_lo) | (wide_msbs(S.meta_hi) << 4))) | (S.imask << 8) | (lane << 16);
        walking = wide_next<kWideShared>(S, top, sh, over, sp, node, err);
      }
      const unsigned m = __ballot_sync(FULL_MASK, lh != 0);
      if (lh) {
        queue[nq + __popc(m & lt)] = make_uint2(lbase, lh);
        pending = true;
      }
      nq += __popc(m);
    }
    const unsigned waiting = __ballot_sync(FULL_MASK, active && !walking && pending);
    const unsigned running = __ballot_sync(FULL_MASK, walking);
    if (nq >= kWideFlush || (waiting && (!running || 32 - __popc(running) >= kWideRefill))) flush();
    if (active && !walking && !pending) {
      const uint32_t prim = !ANY ? (uint32_t)sbest[lane] : (sbest[lane] != ~0ull ? s_bid[wq][lane] : kMiss);
      hits[s_rid[wq][lane]] = wide_result(prim, sbslot[lane]);
      active = false;
    }
  }
}
}  // namespace gprtcu

using namespace gprtcu;


namespace {

struct WideScratch {
  size_t counters, queue, total;
};

WideScratch wide_layout(uint32_t meshes, uint32_t n) {
  WideScratch L;
  size_t off = sizeof(ScratchHeader);
  L.counters = off;
  off += 256;
  L.queue = off;
  off += gprtcu_align256((size_t)n * sizeof(WorkItem));
  L.total = off;
  (void)meshes;
  return L;
}

}  // namespace

extern "C" GPRTCU_API size_t gprtcuWideScratchSize(uint32_t numMeshes, uint32_t totalTriangles) {
  return wide_layout(numMeshes, totalTriangles).total;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuWideBuild(const gprtcuLbvh *binary, const uint32_t *triOffsets,
                                                   uint32_t numMeshes, gprtcuWideBvh *out, void *scratch,
                                                   size_t scratchBytes, gprtcuStream stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!binary || !out || numMeshes == 0) return GPRTCU_ERR_INVALID_ARG;
  const uint32_t n = binary->numPrims;
  if (n == 0 || numMeshes > n || (numMeshes > 1 && !triOffsets)) return GPRTCU_ERR_INVALID_ARG;
  if (!binary->leafTris || (n > numMeshes && !binary->bvh2)) return GPRTCU_ERR_INVALID_ARG;
  if (!out->nodes || !out->leafTris || !out->roots || out->capacity < n) return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)out->nodes & 15) || ((uintptr_t)out->leafTris & 15)) return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  const WideScratch L = wide_layout(numMeshes, n);
  if (scratchBytes < L.total) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  char *s = (char *)scratch;
  GPRTCU_TRY(cudaMemsetAsync(s, 0, L.queue, stream));  // header, counters
  uint32_t *counters = (uint32_t *)(s + L.counters);
  WorkItem *queue = (WorkItem *)(s + L.queue);
  const uint32_t *toff = numMeshes > 1 ? triOffsets : nullptr;
  k_wide_init<<<(numMeshes + 255) / 256, 256, 0, stream>>>(toff, numMeshes, n, queue, out->roots, counters);
  GPRTCU_TRY(cudaGetLastError());
  // The whole-GPU levels are launches whose grid is what fits on the GPU at
  // once (7 CTAs of 128 threads per SM: 72 registers, 24 KB of shared memory):
  // a grid-stride loop with a second wave of CTAs ran the level for about
  // twice a CTA's share (6.6 against 4.8 ms).
  static std::atomic<int> level_ctas_cache{0};  // host threads may race to fill it with the same value
  int level_ctas = level_ctas_cache.load(std::memory_order_relaxed);
  if (!level_ctas) {
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_wide_level<kWideRestForm>, 128, 0) != cudaSuccess || occ < 1)
      occ = 1;
    level_ctas = occ;
    level_ctas_cache.store(occ, std::memory_order_relaxed);
  }
  const int grid = gprtcu_num_sms() * level_ctas;
  auto launch = [&](auto kernel, int ctas, cudaLaunchAttribute at, uint32_t most) -> cudaError_t {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(128);
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, (const Bvh2Node *)binary->bvh2, (const float4 *)binary->leafTris, toff,
                              (WideNode *)out->nodes, (float4 *)out->leafTris, queue, counters, most);
  };
  cudaLaunchAttribute cluster = {}, rest = {};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  rest.id = cudaLaunchAttributeCooperative;
  rest.val.cooperative = 1;
  auto few = [&](uint32_t most) {
    cluster.val.clusterDim.x = kWideCluster;
    return launch(k_wide_level<kWideClusterForm>, kWideCluster, cluster, most);
  };
  auto levels = [&](int count) -> cudaError_t {
    cluster.val.clusterDim.x = 1;
    for (int i = 0; i < count; ++i) {
      const cudaError_t e = launch(k_wide_level<kWideLevelForm>, grid, cluster, 0u);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  };
  // How deep the tree is only the device knows, and a launch that finds its
  // level empty costs 4 us of the stream: with one launch for each of the 62
  // levels that a tree could have, a collapse took 0.31 ms whatever its size.
  // So: the cluster takes the first levels, up to kWideFew items; as many
  // whole-GPU levels follow as scenes of n triangles have needed (8 to 13
  // levels in all for 20,001 to 4.2 M of them, 10 for a batch of 67 M); the
  // cluster goes on while at most kWideMore items are left, which is usually
  // the end; and one launch takes what then is left of a tree that stays wide,
  // or widens again, that late.  Up to 100,000 triangles the cluster alone is
  // no slower than the 62 launches were.
  //   1,501 triangles 0.36 -> 0.06 ms; 20,001 0.31 -> 0.08; 150,001 0.33 ->
  //   0.10; 1 M 0.41 -> 0.19; 4.2 M 0.64 -> 0.43; 67 M in 4,096 meshes 2.97 ->
  //   2.75 ms.  In meshes graded towards a point most levels come late: 1 M /
  //   4.2 M triangles over 25 octaves of distance 0.64 / 0.84 ms with 62
  //   launches, 2.8 / 10.7 with the cluster to end them, 0.50 / 0.69 so.
  int lg = 0;
  while (lg < 32 && (1ull << lg) < n) ++lg;
  if (gprtcu_max_cluster() < kWideCluster) {
    GPRTCU_TRY(launch(k_wide_level<kWideRestForm>, grid, rest, gprtcu_spin_budget()));
  } else if (n > 8192) {
    GPRTCU_TRY(few(kWideFew));
    GPRTCU_TRY(levels(lg > 16 ? lg - 14 : 2));
    GPRTCU_TRY(few(n > 100000 ? kWideMore : UINT32_MAX));
    if (n > 100000) GPRTCU_TRY(launch(k_wide_level<kWideRestForm>, grid, rest, gprtcu_spin_budget()));
  } else {
    GPRTCU_TRY(few(UINT32_MAX));
  }
  if (out->numNodes) GPRTCU_TRY(cudaMemcpyAsync(out->numNodes, counters + C_TAIL, 4, cudaMemcpyDeviceToDevice, stream));
  return GPRTCU_OK;
}

extern "C" GPRTCU_API gprtcuStatus gprtcuWideTrace(const gprtcuWideBvh *bvh, const uint32_t *rayOffsets,
                                                   uint32_t numMeshes, const float *rays, uint64_t numRays, int anyHit,
                                                   gprtcuHit *hits, void *scratch, size_t scratchBytes,
                                                   gprtcuStream stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!bvh || numMeshes == 0 || (numMeshes > 1 && !rayOffsets)) return GPRTCU_ERR_INVALID_ARG;
  if ((!rays || !hits) && numRays) return GPRTCU_ERR_INVALID_ARG;
  if (numRays == 0) return GPRTCU_OK;
  if (!bvh->nodes || !bvh->leafTris || !bvh->roots) return GPRTCU_ERR_INVALID_ARG;
  if (((uintptr_t)rays & 15) || ((uintptr_t)bvh->nodes & 15) || ((uintptr_t)bvh->leafTris & 15))
    return GPRTCU_ERR_INVALID_ARG;
  if (!scratch || ((uintptr_t)scratch & 255)) return GPRTCU_ERR_INVALID_ARG;
  if (scratchBytes < sizeof(ScratchHeader)) return GPRTCU_ERR_SCRATCH_TOO_SMALL;
  ScratchHeader *hdr = (ScratchHeader *)scratch;
  unsigned long long *counter = reinterpret_cast<unsigned long long *>(&hdr->ticket[0]);
  GPRTCU_TRY(cudaMemsetAsync(scratch, 0, sizeof(ScratchHeader), stream));
  const int blocks = gprtcu_num_sms() * kWideCtas;
  const uint64_t need = (numRays + kWideThreads - 1) / kWideThreads;
  const int grid = (int)(need < (uint64_t)blocks ? need : blocks);
  auto launch = [&](auto kernel) {
    kernel<<<grid, kWideThreads, 0, stream>>>((const WideNode *)bvh->nodes, (const float4 *)bvh->leafTris, bvh->roots,
                                              rayOffsets, numMeshes, (const float4 *)rays, numRays, (Hit *)hits,
                                              counter, &hdr->status);
  };
  auto pick = [&](auto v8) {
    constexpr bool V = decltype(v8)::value;
    if (numMeshes > 1) anyHit ? launch(k_trace_wide<true, true, V>) : launch(k_trace_wide<false, true, V>);
    else anyHit ? launch(k_trace_wide<true, false, V>) : launch(k_trace_wide<false, false, V>);
  };
  if (((uintptr_t)bvh->nodes & 31) == 0) pick(std::true_type());
  else pick(std::false_type());
  GPRTCU_TRY(cudaGetLastError());
  const uint64_t need_r = (numRays + kRefineThreads - 1) / kRefineThreads;
  const int grid_r = (int)(need_r < (uint64_t)gprtcu_num_sms() * 4 ? need_r : gprtcu_num_sms() * 4);
  k_wide_refine<<<grid_r, kRefineThreads, 0, stream>>>((const float4 *)bvh->leafTris, (const float4 *)rays,
                                                       numRays, (Hit *)hits);
  GPRTCU_TRY(cudaGetLastError());
  return GPRTCU_OK;
}
