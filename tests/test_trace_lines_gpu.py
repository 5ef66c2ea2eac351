"""The ray counts at which a traversal changes its form: the same hits on both
sides of each line, and no step in time at the line of the shared-visit form
that goes up as more rays come."""
import numpy as np
import pytest

import oracle
from gprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _line(sixths):
    """The largest ray count of the shared-visit form: that many sixths of 16
    rays for each of 12 x 2 warps per SM."""
    return _sms() * 12 * 2 * 16 * sixths // 6


def _bits(h):
    return h.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n,sixths", [(2047, 6), (2048, 9)])
def test_triangle_line(cuda, n, sixths):
    import torch
    from gprt_b200 import api
    m = _line(sixths)
    pos, tri = scenes.soup(n, seed=n, sigma=0.03)
    rays_h = scenes.rays(m + 1, seed=n)
    rays = torch.from_numpy(rays_h).cuda()
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    below, above = _bits(api.trace(b, rays[:m])), _bits(api.trace(b, rays))
    assert np.array_equal(below, above[:m])
    exp = oracle.trace_lbvh(pos, tri, oracle.lbvh_build_tri(pos, tri), rays_h[-3000:])
    assert np.array_equal(above[-3000:, 0], exp["prim"])


@pytest.mark.parametrize("n,sixths", [(100000, 16), (100001, 12)])
@pytest.mark.parametrize("kind", ["spheres", "lss"])
def test_prim_line(cuda, n, sixths, kind):
    import torch
    from gprt_b200 import api
    m = _line(sixths)
    rng = np.random.default_rng(n)
    v = np.concatenate([rng.random((n + 1, 3)), rng.uniform(0.001, 0.004, (n + 1, 1))], 1).astype(np.float32)
    v[1::2, :3] = v[:-1:2, :3][:len(v[1::2])] + rng.normal(0, 0.004, (len(v[1::2]), 3)).astype(np.float32)
    idx = np.stack([np.arange(n) & ~1, (np.arange(n) & ~1) + 1], 1).astype(np.uint32) % (n + 1)
    rays_h = scenes.rays(m + 1, seed=n)
    rays, vt, it = torch.from_numpy(rays_h).cuda(), torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    if kind == "spheres":
        b = api.lbvh_build_boxes(api.sphere_bounds(vt[:n]))
        run = lambda r, u: api.trace_spheres(b, vt[:n], r, u=u)
    else:
        b = api.lbvh_build_boxes(api.lss_bounds(vt, it))
        run = lambda r, u: api.trace_lss(b, vt, it, r, u=u)
    u = [torch.zeros(m + 1, device="cuda") for _ in range(2)]
    below, above = _bits(run(rays[:m], u[0])), _bits(run(rays, u[1]))
    assert np.array_equal(below, above[:m])
    assert torch.equal(u[0][:m].view(torch.int32), u[1][:m].view(torch.int32))
    e = oracle.trace_user_brute(0 if kind == "spheres" else 1, v[:n] if kind == "spheres" else v, rays_h[-300:],
                                *(() if kind == "spheres" else (idx,)))
    assert np.array_equal(above[-300:, 0], e["prim"])


@pytest.mark.parametrize("n", [1, 2, 5000])
def test_any_hit_whatever_the_rays(cuda, n):
    """An any-hit call reports the first hit of the near-first walk, so the
    same one however many rays the call has and however they share warps."""
    import torch
    from gprt_b200 import api
    pos, tri = scenes.soup(n, seed=n + 3, sigma=0.1)
    rays = torch.from_numpy(scenes.rays(200003, seed=n)).cuda()
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    sph = torch.from_numpy(np.concatenate([np.random.default_rng(n).random((n + 1, 3)), np.full((n + 1, 1), 0.04)],
                                          1).astype(np.float32)).cuda()
    idx = torch.stack([torch.arange(n), torch.arange(n) + 1], 1).int().cuda()
    bs, bl = api.lbvh_build_boxes(api.sphere_bounds(sph[:n])), api.lbvh_build_boxes(api.lss_bounds(sph, idx))
    runs = [lambda r, u: api.trace(b, r, anyhit=True),
            lambda r, u: api.trace_spheres(bs, sph[:n], r, u=u, anyhit=True),
            lambda r, u: api.trace_lss(bl, sph, idx, r, u=u, anyhit=True)]
    for run in runs:
        u = torch.zeros(200003, device="cuda")
        full = _bits(run(rays, u)).copy()
        for m in (1, 33, 700, 4099, 30011, 56001):
            v = torch.zeros(m, device="cuda")
            assert np.array_equal(_bits(run(rays[:m], v)), full[:m])
            assert torch.equal(v.view(torch.int32), u[:m].view(torch.int32))


def test_no_step_at_the_line(cuda):
    """Spheres, around twice 16 rays for every warp that fits, where the lane
    per ray takes over: a call with a few more rays does not take clearly
    longer, nor does one with fewer."""
    import torch
    from gprt_b200 import api
    n, m, slack = 1_000_001, _line(12), 1.2
    a, b = int(m * 0.994), int(m * 1.012)
    rays = api.gen_rays(b, seed=5)
    s = torch.rand((n, 4), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    s[:, 3].mul_(0.0015).add_(0.0005)
    t = api.lbvh_build_boxes(api.sphere_bounds(s))
    hits, scr = torch.empty((b, 2), dtype=torch.int32, device="cuda"), api.scratch(256)

    def us(r):
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                api.trace_spheres(t, s, r, hits=hits[:r.shape[0]], scr=scr)
            e[1].record()
            e[1].synchronize()
            times.append(1e2 * e[0].elapsed_time(e[1]))
        return sorted(times[2:])[3]

    below, above = us(rays[:a]), us(rays)
    assert above < slack * below and below < slack * above, (below, above)


def _scene(kind, n, reach=0.0):
    """n primitives apart from each other (as strands), or within `reach`."""
    rng = np.random.default_rng(n)
    v = np.concatenate([rng.random((n + 1, 3)), rng.uniform(0.0005, 0.002 + reach, (n + 1, 1))], 1).astype(np.float32)
    v[1::2, :3] = v[:-1:2, :3][:len(v[1::2])] + rng.normal(0, 0.004 + reach, (len(v[1::2]), 3)).astype(np.float32)
    idx = np.stack([np.arange(n) & ~1, (np.arange(n) & ~1) + 1], 1).astype(np.uint32) % (n + 1)
    return (v[:n] if kind == "spheres" else v), idx


def _runner(kind, v, idx):
    import torch
    from gprt_b200 import api
    vt, it = torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    if kind == "spheres":
        b = api.lbvh_build_boxes(api.sphere_bounds(vt))
        return lambda r, **k: api.trace_spheres(b, vt, r, **k)
    b = api.lbvh_build_boxes(api.lss_bounds(vt, it))
    return lambda r, **k: api.trace_lss(b, vt, it, r, **k)


@pytest.mark.parametrize("reach", [0.0, 0.1])
@pytest.mark.parametrize("n", [1, 2, 2047, 2048, 8191, 8192, 16383])
@pytest.mark.parametrize("kind", ["spheres", "lss"])
def test_few_prims_lines(cuda, kind, n, reach):
    """Few primitives: the same hits and u on both sides of each ray count
    where the form changes, exit hits too, and the oracle's primitives."""
    import torch
    v, idx = _scene(kind, n, reach)
    run = _runner(kind, v, idx)
    lines = [_line(6), _line(9), _sms() * 8 * 128]
    m = lines[-1] + 1
    rays_h = scenes.rays(m, seed=n)
    rays_h[::97, 7] = np.nan
    rays_h[5::97, 3] = -1.0
    rays = torch.from_numpy(rays_h).cuda()
    for exit_test in (False, True):
        u = torch.zeros(m, device="cuda")
        full = _bits(run(rays, u=u, exit_test=exit_test)).copy()
        for k in (1, 4099, lines[0], lines[0] + 1, lines[1], lines[1] + 1, lines[2]):
            w = torch.zeros(k, device="cuda")
            assert np.array_equal(_bits(run(rays[:k], u=w, exit_test=exit_test)), full[:k])
            assert torch.equal(w.view(torch.int32), u[:k].view(torch.int32))
        if not exit_test:
            ok = np.arange(m - 300, m)[~np.isnan(rays_h[-300:, 7])]
            e = oracle.trace_user_brute(0 if kind == "spheres" else 1, v, rays_h[ok],
                                        *(() if kind == "spheres" else (idx,)))
            assert np.array_equal(full[ok, 0], e["prim"])


@pytest.mark.parametrize("kind,n,m", [("spheres", 1001, 130001), ("lss", 1001, 130001), ("lss", 101, 1000001)])
def test_few_prims_take_no_longer_than_any_hit(cuda, kind, n, m):
    """Few primitives that lie apart, which most rays miss: a closest hit has
    little more to do than an any hit."""
    import torch
    from gprt_b200 import api
    run, rays = _runner(kind, *_scene(kind, n)), api.gen_rays(m, seed=5)
    hits, scr = torch.empty((m, 2), dtype=torch.int32, device="cuda"), api.scratch(256)

    def us(any_hit):
        times = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(20):
                run(rays, hits=hits, scr=scr, anyhit=any_hit)
            e[1].record()
            e[1].synchronize()
            times.append(50.0 * e[0].elapsed_time(e[1]))
        return sorted(times[2:])[3]

    assert us(False) < 1.15 * us(True)
