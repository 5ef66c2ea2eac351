"""The collapse at the sizes where its sequence of launches changes (one cluster
for all levels; cluster, whole-GPU levels, cluster; and again), on ordinary
scenes and on one whose tree is narrow for many levels before it widens.
Every wide node but the roots is the child of one node, every triangle in one
leaf, and the hits are those of the binary tree."""
import numpy as np
import pytest

from gprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _late(n, levels=10):
    """Large triangles around a corner at halving distances, all others in
    the corner: what covers the corner is small beside its siblings, so wide
    nodes take it apart late."""
    rng = np.random.default_rng(n)
    pos, tri = scenes.soup(n, seed=n, sigma=1e-6)
    pos = pos * np.float32(2.0**-levels)
    k = np.repeat(np.arange(levels), 64)
    c = rng.uniform(0.5, 1.0, (k.size, 1, 3)) * (2.0**-k)[:, None, None]
    d = np.float32(rng.normal(0, 0.3, (k.size, 1, 3)) * (2.0**-k)[:, None, None])
    pos[:3 * k.size] = np.concatenate([c - d, c, c + d], 1).reshape(-1, 3).astype(np.float32)
    return pos.astype(np.float32), tri


@pytest.mark.parametrize("n,late", [(700, 0), (8192, 0), (8193, 0), (8193, 1), (100000, 0), (100001, 0), (100001, 1),
                                    (400000, 1)])
def test_wide_collapse_launches(cuda, n, late):
    import torch
    from gprt_b200 import api
    pos, tri = _late(n) if late else scenes.soup(n, seed=n, sigma=0.01)
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    w = api.wide_build(b)
    d = api.wide_decode(w)
    used = d["meta"] != 0xFF
    inner = used & (((d["imask"][:, None] >> np.arange(8)) & 1) == 1)
    nodes = (d["child_base"][:, None].astype(np.int64) + d["meta"])[inner]
    leaves = (d["leaf_base"][:, None].astype(np.int64) + d["meta"])[used & ~inner]
    assert np.array_equal(np.sort(nodes), np.arange(1, d["count"]))
    assert np.array_equal(np.sort(leaves), np.arange(n))
    assert np.array_equal(np.sort(d["leaf"][:, 3].view(np.uint32)), np.arange(n, dtype=np.uint32))
    rays = torch.from_numpy(scenes.rays(3000, seed=n)).cuda()
    hw, hb = api.hits_numpy(api.wide_trace(w, rays)), api.hits_numpy(api.trace(b, rays))
    assert np.array_equal(hw["prim"], hb["prim"]) and np.array_equal(hw["t"].view(np.uint32), hb["t"].view(np.uint32))
