// lbvh.cuh -- device-side layouts of the LBVH traversal data.
#pragma once
#include <stdint.h>

namespace gprtcu {

// One inner node of the binary traversal layout: both child boxes and both
// child references in 64 bytes, one 32-byte half per child, so that a half is
// one load.  box is the child's {lo.x, lo.y, hi.x, hi.y, lo.z, hi.z} -- the
// order in which a ray's origin and reciprocal direction take four register
// pairs for packed arithmetic: (x, y) twice and (z, z) --; ref >= 0 is an
// inner node, ref < 0 is leaf slot ~ref (the leaf's position in sorted order).
struct __align__(16) Bvh2Child {
  float box[6];
  int ref;
  int pad;
};
struct __align__(16) Bvh2Node {
  Bvh2Child c[2];
};
static_assert(sizeof(Bvh2Node) == 64, "64-byte node");
// Word of Bvh2Child::box that holds component k of {lo.xyz, hi.xyz}.
__host__ __device__ constexpr int box_word(int k) { return k == 2 ? 4 : (k == 3 ? 2 : (k == 4 ? 3 : k)); }

// Triangle of leaf slot s: three float4 {v.xyz, w}; w of the first holds the
// primitive id bits.
struct Hit {
  uint32_t prim;
  float t;
};

}  // namespace gprtcu
