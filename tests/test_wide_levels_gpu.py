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


def _check(api, w, n):
    """Every wide node but the root is the child of one node, every triangle
    in one leaf."""
    d = api.wide_decode(w)
    used = d["meta"] != 0xFF
    inner = used & (((d["imask"][:, None] >> np.arange(8)) & 1) == 1)
    nodes = (d["child_base"][:, None].astype(np.int64) + d["meta"])[inner]
    leaves = (d["leaf_base"][:, None].astype(np.int64) + d["meta"])[used & ~inner]
    assert np.array_equal(np.sort(nodes), np.arange(1, d["count"]))
    assert np.array_equal(np.sort(leaves), np.arange(n))
    assert np.array_equal(np.sort(d["leaf"][:, 3].view(np.uint32)), np.arange(n, dtype=np.uint32))


def _graded(n):
    """A mesh graded towards a point: distances from it log-uniform over 25
    octaves, sizes alike, so levels stay wide far down the tree."""
    rng = np.random.default_rng(n)
    k = 2.0**(-25 * rng.random((n, 1)))
    c = (rng.random((n, 3)) * k)[:, None, :]
    pos = (c + rng.normal(0, 0.01, (n, 3, 3)) * k[:, None, :]).reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


def test_wide_collapse_graded(cuda):
    """As above on a graded mesh, whose levels past the first dozen the last
    launch takes together; and it takes less time than four builds of the tree (ten
    with one cluster for them)."""
    import torch
    from gprt_b200 import api
    n = 1_000_001
    pos, tri = _graded(n)
    p, t = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda()
    b, w = api.Lbvh(n), api.WideBvh(n)

    def us(f):
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            f()
            e[1].record()
            e[1].synchronize()
            times.append(1e3 * e[0].elapsed_time(e[1]))
        return sorted(times[2:])[3]

    build = us(lambda: api.lbvh_build_triangles(p, t, b))
    collapse = us(lambda: api.wide_build(b, wide=w))
    _check(api, w, n)
    rays = torch.from_numpy(scenes.rays(3000, seed=n)).cuda()
    hw, hb = api.hits_numpy(api.wide_trace(w, rays)), api.hits_numpy(api.trace(b, rays))
    assert np.array_equal(hw["prim"], hb["prim"]) and np.array_equal(hw["t"].view(np.uint32), hb["t"].view(np.uint32))
    assert api.scratch_status(w.scratch) == 0
    assert collapse < 4 * build, (collapse, build)


@pytest.mark.parametrize("n", [700, 50_000, 200_001])
def test_wide_collapse_captured(cuda, n):
    """A captured collapse (its launches carry cluster and cooperative
    attributes) gives the same nodes for new vertices at each replay."""
    import torch
    from gprt_b200 import api
    pos, tri = _graded(n)
    p, t = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda()
    b, w = api.Lbvh(n), api.WideBvh(n)
    run = lambda: api.wide_build(api.lbvh_build_triangles(p, t, b), wide=w)
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    rays = torch.from_numpy(scenes.rays(3000, seed=n)).cuda()
    for step in range(2):
        p.copy_(torch.from_numpy(pos)[torch.randperm(3 * n, generator=torch.Generator().manual_seed(step))] if step else
                torch.from_numpy(pos))
        w.nodes.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _check(api, w, n)
        assert torch.equal(api.wide_trace(w, rays), api.trace(b, rays))
