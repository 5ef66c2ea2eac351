"""Binary traversal over the forms its launch rule tells apart: few rays (spread
over the warps, fewer than 32 to a warp) up to full warps with a ragged end,
traversal nodes on 32-byte boundaries or only on 16-byte ones, one mesh or a
batch with one-triangle meshes; and a refit into nodes that are only 8-byte
aligned.  Ids and t bits equal the oracle's traversal of the same tree."""
import numpy as np
import pytest

import oracle
from gprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _shift_nodes(bvh, nbytes):
    """Moves the traversal nodes to `nbytes` past a 256-byte boundary."""
    import torch
    words = bvh.bvh2.numel()
    buf = torch.zeros(words + 64, dtype=torch.float32, device="cuda")
    assert buf.data_ptr() % 256 == 0
    k = nbytes // 4
    bvh.bvh2 = buf[k:k + words].view(-1, 16)
    bvh.desc.bvh2 = bvh.bvh2.data_ptr()


def _expect(pos, tri, rays):
    return oracle.trace_lbvh(pos, tri, oracle.lbvh_build_tri(pos, tri), rays)


def _same(got, exp):
    hit = exp["prim"] != 0xFFFFFFFF
    return np.array_equal(got["prim"], exp["prim"]) and np.array_equal(got["t"][hit].view(np.uint32),
                                                                       exp["t"][hit].view(np.uint32))


@pytest.mark.parametrize("shift", [0, 16, 32])
@pytest.mark.parametrize("n,m", [(1, 3), (2, 1), (3, 33), (700, 4099), (5000, 18943), (5000, 18945), (20000, 200003)])
def test_trace_forms(cuda, n, m, shift):
    import torch
    from gprt_b200 import api
    pos, tri = scenes.soup(n, seed=n + m, sigma=0.02 if n > 100 else 0.3)
    rays = scenes.rays(m, seed=m)
    p, t, r = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda(), torch.from_numpy(rays).cuda()
    b = api.Lbvh(n)
    _shift_nodes(b, shift)
    api.lbvh_build_triangles(p, t, b)
    exp = _expect(pos, tri, rays)
    assert _same(api.hits_numpy(api.trace(b, r)), exp)
    anyh = api.hits_numpy(api.trace(b, r, anyhit=True))
    assert np.array_equal(anyh["prim"] != 0xFFFFFFFF, exp["prim"] != 0xFFFFFFFF)


@pytest.mark.parametrize("n,m", [(40, 700), (5000, 300), (60000, 64)])
def test_trace_overlapping(cuda, n, m):
    """Triangles as large as the scene: nearly every box is entered, and the
    shared stack of the few-ray form fills up."""
    import torch
    from gprt_b200 import api
    pos, tri = scenes.soup(n, seed=3, sigma=1.0)
    rays = scenes.rays(m, seed=4)
    rays[::3, 7] = 0.9
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    assert _same(api.hits_numpy(api.trace(b, torch.from_numpy(rays).cuda())), _expect(pos, tri, rays))


@pytest.mark.parametrize("n", [5000000, 5000001, 12000001])
@pytest.mark.parametrize("anyhit", [False, True])
def test_trace_large_meshes(cuda, n, anyhit):
    """The sizes at which a warp's refill changes; the hits of the quantised
    traversal, whose code does not depend on the size."""
    from gprt_b200 import api
    pos, tri = api.gen_mixture(n, clusters=64, seed=9)
    rays = api.gen_rays(200001, seed=10)
    b = api.lbvh_build_triangles(pos, tri, api.Lbvh(n, with_aabbs=False))
    hb = api.hits_numpy(api.trace(b, rays, anyhit=anyhit))
    hw = api.hits_numpy(api.wide_trace(api.wide_build(b), rays, anyhit=anyhit))
    if anyhit:
        assert np.array_equal(hb["prim"] != 0xFFFFFFFF, hw["prim"] != 0xFFFFFFFF)
    else:
        assert np.array_equal(hb["prim"], hw["prim"]) and np.array_equal(hb["t"].view(np.uint32), hw["t"].view(np.uint32))


@pytest.mark.parametrize("shift", [0, 16])
def test_batch_trace_forms(cuda, shift):
    import torch
    from gprt_b200 import api
    sizes = [1, 700, 1, 1, 33, 2, 4000]
    off = np.concatenate([[0], np.cumsum(sizes)])
    pos, tri = scenes.soup(int(off[-1]), seed=4, sigma=0.05)
    rays = scenes.rays(int(off[-1]) * 3, seed=5)
    roff = off * 3
    b = api.BatchLbvh(off)
    _shift_nodes(b, shift)
    api.batch_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda(), b)
    ro = torch.from_numpy(roff.astype(np.int32)).cuda()
    got = api.hits_numpy(api.batch_trace(b, torch.from_numpy(rays).cuda(), ro))
    for k in range(len(sizes)):
        t = np.ascontiguousarray(tri[off[k]:off[k + 1]])
        assert _same(got[roff[k]:roff[k + 1]], _expect(pos, t, rays[roff[k]:roff[k + 1]])), k


@pytest.mark.parametrize("shift", [0, 8, 16])
def test_refit_node_alignment(cuda, shift):
    """A refit writes the same traversal nodes wherever they lie."""
    import torch
    from gprt_b200 import api
    n = 3001
    pos, tri = scenes.soup(n, seed=8, sigma=0.05)
    p, t = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda()
    b = api.lbvh_build_triangles(p, t)
    want = api.lbvh_refit_triangles(p * 0.5 + 0.1, t, b).bvh2.clone()
    api.lbvh_refit_triangles(p, t, b)
    keep = b.bvh2.clone()
    _shift_nodes(b, shift)
    b.bvh2.copy_(keep)
    api.lbvh_refit_triangles(p * 0.5 + 0.1, t, b)
    assert torch.equal(b.bvh2.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("anyhit", [False, True])
def test_instance_node_alignment(cuda, anyhit):
    """Instanced traversal gives the same hits wherever the nodes of the two
    levels lie (mesh sizes include one triangle, a deep mix of levels)."""
    import torch
    from gprt_b200 import api
    rng = np.random.default_rng(3)
    sizes = [1, 900, 40, 1, 5000]
    off = np.concatenate([[0], np.cumsum(sizes)])
    pos, tri = scenes.soup(int(off[-1]), seed=6, sigma=0.05)
    p, t = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda()
    n = 300
    rec = np.zeros(n, np.dtype(api.INSTANCE_DTYPE))
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    m = np.concatenate([q * rng.uniform(0.5, 1.5, (n, 1, 1)), rng.uniform(0, 4, (n, 3, 1))], 2)
    rec["transform"] = m.reshape(n, 12)
    rec["custom_mask"] = 0xFF << 24
    rec["blas"] = np.arange(n) % len(sizes)
    rays = torch.from_numpy(scenes.rays(20011, seed=9) * np.array([4, 4, 4, 1, 1, 1, 1, 1], np.float32)).cuda()
    out = []
    for shift in (0, 16):
        b = api.BatchLbvh(off)
        _shift_nodes(b, shift)
        api.batch_build_triangles(p, t, b)
        tlas = api.Tlas(api.instances_tensor(rec), b.root, len(sizes))
        _shift_nodes(tlas.bvh, shift)
        tlas.build()
        h, i = api.trace_instances(tlas, b, rays, b.tri_off, len(sizes), anyhit=anyhit)
        out.append((h.clone(), i.clone()))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert int((out[0][1] >= 0).sum()) > 100


@pytest.mark.parametrize("m", [1, 37, 4099, 151553])
def test_prims_forms(cuda, m):
    """Spheres and swept spheres: few to many rays, nodes on 16-byte
    boundaries; against the oracle's search over every primitive where that is
    small, else against the 32-byte form."""
    import torch
    from gprt_b200 import api
    n = 300 if m < 5000 else 20000
    rng = np.random.default_rng(m)
    v = np.concatenate([rng.random((n + 1, 3)), rng.uniform(0.002, 0.02, (n + 1, 1))], 1).astype(np.float32)
    idx = np.stack([np.arange(n), np.arange(n) + 1], 1).astype(np.uint32)
    v[:, :3] = np.cumsum(np.vstack([v[:1, :3], rng.normal(0, 0.03, (n, 3))]), 0) % 1.0
    vt, it = torch.from_numpy(v.astype(np.float32)).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    rays_h = scenes.rays(m, seed=m)
    rays = torch.from_numpy(rays_h).cuda()
    for kind in (0, 1):
        out = []
        for shift in (0, 16):
            b = api.Lbvh(n)
            _shift_nodes(b, shift)
            api.lbvh_build_boxes(api.sphere_bounds(vt[:n]) if kind == 0 else api.lss_bounds(vt, it), b)
            u = torch.zeros(m, device="cuda")
            h = api.trace_spheres(b, vt[:n], rays, u=u) if kind == 0 else api.trace_lss(b, vt, it, rays, u=u)
            a = api.trace_spheres(b, vt[:n], rays, anyhit=True) if kind == 0 else api.trace_lss(b, vt, it, rays,
                                                                                              anyhit=True)
            assert torch.equal(a[:, 0] == -1, h[:, 0] == -1)
            out.append((api.hits_numpy(h), u.cpu().numpy()))
        (h0, u0), (h1, u1) = out
        assert np.array_equal(h0["prim"], h1["prim"]) and np.array_equal(h0["t"].view(np.uint32),
                                                                        h1["t"].view(np.uint32))
        assert np.array_equal(u0.view(np.uint32), u1.view(np.uint32))
        if n == 300:
            e = oracle.trace_user_brute(kind, v[:n] if kind == 0 else v, rays_h, *(() if kind == 0 else (idx,)))
            assert np.array_equal(h0["prim"], e["prim"])


def _odd_rays(m, seed, share):
    """Rays with some components infinite, NaN, zero or huge."""
    rng = np.random.default_rng(seed)
    rays = scenes.rays(m, seed=seed)
    odd = np.float32([np.nan, np.inf, -np.inf, 0.0, -0.0, -1.0, 1e30, -1e30, 1e-40, 3.4e38])
    rays = np.where(rng.random((m, 8)) < share, odd[rng.integers(0, odd.size, (m, 8))], rays).astype(np.float32)
    rays[::97, 4:7] = 0.0  # no direction
    return rays


@pytest.mark.parametrize("n", [1, 300])
def test_prims_odd_rays(cuda, n):
    """Rays whose primitive tests can give a distance that is no number: such
    a hit counts if it is the ray's first.  One primitive: as the oracle says;
    more: the same however many rays the call has."""
    import torch
    from gprt_b200 import api
    few, many = 4099, 151553
    rng = np.random.default_rng(n)
    v = np.concatenate([rng.random((n + 1, 3)), rng.uniform(0.1, 0.3, (n + 1, 1))], 1).astype(np.float32)
    idx = np.stack([np.arange(n), np.arange(n) + 1], 1).astype(np.uint32)
    vt, it = torch.from_numpy(v).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    rays_h = _odd_rays(many, n, 0.05)
    rays = torch.from_numpy(rays_h).cuda()
    for kind in (0, 1):
        b = api.lbvh_build_boxes(api.sphere_bounds(vt[:n]) if kind == 0 else api.lss_bounds(vt, it))
        run = (lambda r, **k: api.hits_numpy(api.trace_spheres(b, vt[:n], r, **k))) if kind == 0 else \
            (lambda r, **k: api.hits_numpy(api.trace_lss(b, vt, it, r, **k)))
        u = torch.zeros(many, device="cuda"), torch.zeros(few, device="cuda")
        full, part, anyh = run(rays, u=u[0]), run(rays[:few].contiguous(), u=u[1]), run(rays, anyhit=True)
        assert np.isnan(full["t"]).sum() > 50
        assert np.array_equal(full[:few].view(np.uint32), part.view(np.uint32))
        assert torch.equal(u[0][:few].view(torch.int32), u[1].view(torch.int32))
        assert np.array_equal(full["prim"] == 0xFFFFFFFF, anyh["prim"] == 0xFFFFFFFF)
        if n == 1:
            e = oracle.trace_user_brute(kind, v[:n] if kind == 0 else v, rays_h, *(() if kind == 0 else (idx,)))
            hit = full["prim"] == 0  # the box test may drop a ray that the primitive test alone would not
            assert np.all(e["prim"][hit] == 0)
            assert np.array_equal(np.isnan(full["t"][hit]), np.isnan(e["t"][hit]))


@pytest.mark.parametrize("stride", [32, 36, 48])
@pytest.mark.parametrize("shift", [0, 16])
def test_solid_forms(cuda, stride, shift):
    """Point location with every cell type, index records on 16-byte
    boundaries or not, nodes likewise, and few to many points: the answers of
    the default layout, a sample of them equal to the oracle's search."""
    import torch
    from gprt_b200 import api
    verts, idx, types = scenes.solid_grid(7, seed=2)
    n = types.size
    wide = np.full((n, stride // 4), 0xFFFFFFFF, np.uint32)
    wide[:, :8] = idx
    vt, tt = torch.from_numpy(verts).cuda(), torch.from_numpy(types).cuda()
    std = api.Solids(vt, torch.from_numpy(idx.view(np.int32)).cuda(), tt)
    alt = api.Solids(vt, torch.from_numpy(wide.view(np.int32)).cuda(), tt)
    alt.desc.indexStride = stride
    for m in (1, 9, 70, 60001):
        pts_h = np.random.default_rng(m).random((m, 4), dtype=np.float32) * 1.1 - 0.05
        pts = torch.from_numpy(pts_h).cuda()
        out = []
        for sol, sh in ((std, 0), (alt, shift)):
            b = api.Lbvh(n)
            _shift_nodes(b, sh)
            api.lbvh_build_boxes(api.solid_bounds(sol)[1], b)
            out.append(api.locate_solid_points(b, sol, pts))
        assert torch.equal(out[0][0], out[1][0])
        assert torch.equal(out[0][1].view(torch.int32), out[1][1].view(torch.int32))
        if m == 70:
            ec, ek, er = oracle.solid_locate_brute(verts, idx, types, pts_h)
            got = out[0][0].cpu().numpy().view(np.uint32)
            assert np.array_equal(got[:, 0], ec) and np.array_equal(got[:, 1], ek)
            assert np.array_equal(out[0][1].cpu().numpy().view(np.uint32), er.view(np.uint32))


@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e9, 1e18])
def test_solid_degenerate_cells(cuda, scale):
    """Cells on which the inversion misbehaves -- random vertices (tangled,
    inverted), repeated and collinear ones, magnitudes at which products
    overflow or vanish -- get the oracle's answers bit for bit."""
    import torch
    from gprt_b200 import api
    rng = np.random.default_rng(5)
    kinds = np.array([10, 14, 13, 12, 23], np.uint8)
    n = 400
    types = kinds[np.arange(n) % 5]
    verts = np.concatenate([rng.random((8 * n, 3)), rng.normal(size=(8 * n, 1))], 1)
    cells = verts.reshape(n, 8, 4)
    cells[::7, 1] = cells[::7, 0]
    cells[1::7, 2:, :3] = cells[1::7, :1, :3] + rng.random((len(cells[1::7]), 6, 1)) * (cells[1::7, 1:2, :3] -
                                                                                      cells[1::7, :1, :3])
    cells[2::7, :, 2] = 0.5
    cells[3::7, :4] = np.round(cells[3::7, :4])
    verts[:, :3] *= scale
    verts = verts.astype(np.float32)
    idx = np.arange(8 * n, dtype=np.uint32).reshape(n, 8)
    pts = np.zeros((3000, 4), np.float32)
    pts[:, :3] = rng.random((3000, 3)) * scale
    pts[:200, :3] = verts[rng.choice(8 * n, 200), :3]
    sol = api.Solids(torch.from_numpy(verts).cuda(), torch.from_numpy(idx.view(np.int32)).cuda(),
                     torch.from_numpy(types).cuda())
    hits, rstw = api.locate_solid_points(api.lbvh_build_boxes(api.solid_bounds(sol)[1]), sol, torch.from_numpy(pts).cuda())
    ec, ek, er = oracle.solid_locate_brute(verts, idx, types, pts)
    got = hits.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[:, 0], ec) and np.array_equal(got[:, 1], ek)
    assert np.array_equal(rstw.cpu().numpy().view(np.uint32), er.view(np.uint32))


@pytest.mark.parametrize("shift", [0, 16, 32])
@pytest.mark.parametrize("n,m", [(1, 5), (2, 40), (9, 100), (3000, 4099), (20000, 100003)])
def test_wide_forms(cuda, n, m, shift):
    """Quantised traversal with its nodes on 32-byte boundaries or only on
    16-byte ones, from one triangle up, rays inside and outside the box: the
    oracle's hits; occlusion likewise."""
    import torch
    from gprt_b200 import api
    pos, tri = scenes.soup(n, seed=n, sigma=0.02 if n > 100 else 0.3)
    rays_h = scenes.rays(m, seed=m + 1)
    rays_h[m // 2:, :3] = np.random.default_rng(m).random((m - m // 2, 3), dtype=np.float32)
    rays_h[::5, 3] = 0.25
    rays_h[1::5, 7] = 1.5
    rays = torch.from_numpy(rays_h).cuda()
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    w = api.WideBvh(n)
    buf = torch.zeros(20 * n + 64, dtype=torch.int32, device="cuda")
    w.nodes = buf[shift // 4:shift // 4 + 20 * n].view(n, 20)
    w.desc.nodes = w.nodes.data_ptr()
    api.wide_build(b, wide=w)
    exp = _expect(pos, tri, rays_h)
    assert _same(api.hits_numpy(api.wide_trace(w, rays)), exp)
    anyh = api.hits_numpy(api.wide_trace(w, rays, anyhit=True))
    assert np.array_equal(anyh["prim"] != 0xFFFFFFFF, exp["prim"] != 0xFFFFFFFF)


@pytest.mark.parametrize("m", [300, 4099, 200003])
def test_ranges_behind_the_origin(cuda, m):
    """Rays whose whole range [tmin, tmax] is negative: the closest hit is
    looked for as any hit is."""
    import torch
    from gprt_b200 import api
    n = 700
    pos, tri = scenes.soup(n, seed=1, sigma=0.05)
    rays = scenes.rays(m, seed=m)
    rays[:, 4:7] *= -1.0
    rays[:, 3] = -4.0
    rays[:, 7] = -0.125
    p, t, r = torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda(), torch.from_numpy(rays).cuda()
    b = api.lbvh_build_triangles(p, t)
    exp = _expect(pos, tri, rays)
    hit = exp["prim"] != 0xFFFFFFFF
    assert hit.sum() > m // 10
    assert _same(api.hits_numpy(api.trace(b, r)), exp)
    assert np.array_equal(api.hits_numpy(api.trace(b, r, anyhit=True))["prim"] != 0xFFFFFFFF, hit)
    rec = np.zeros(3, np.dtype(api.INSTANCE_DTYPE))
    rec["transform"][:, [0, 5, 10]] = 1.0
    rec["transform"][:, 3] = [0.0, 50.0, 100.0]
    rec["custom_mask"] = 0xFF << 24
    h, i = api.trace_instances(api.Tlas(api.instances_tensor(rec), b.root, 1), b, r)
    assert np.array_equal(api.hits_numpy(h)["prim"], exp["prim"])
    sph = np.concatenate([np.random.default_rng(2).random((n, 3)), np.full((n, 1), 0.03)], 1).astype(np.float32)
    s = torch.from_numpy(sph).cuda()
    got = api.hits_numpy(api.trace_spheres(api.lbvh_build_boxes(api.sphere_bounds(s)), s, r))
    e = oracle.trace_user_brute(0, sph, rays)
    assert np.array_equal(got["prim"], e["prim"]) and (e["prim"] != 0xFFFFFFFF).sum() > m // 10


@pytest.mark.parametrize("scale", [1.0, 1e14])
def test_prims_odd_prims(cuda, scale):
    """Swept spheres that reach so far that squares overflow and a test's
    distance is no number (or, at 1e14 with directions as long, where every
    test's is).  Such a hit counts if it is the ray's first in near-first
    order: one lies behind ordinary ones but in the nearer half of the tree.
    The same hits however many rays the call has."""
    import torch
    from gprt_b200 import api
    few, many = 100003, 300007
    rng = np.random.default_rng(11)
    far = 1e20 if scale == 1.0 else 60.0
    v = np.zeros((522, 4))
    v[0::2, 0] = 10.0 + 0.1 * np.arange(261)  # 256 that reach far, all from x = 10 on
    v[1::2, 0] = far
    v[0, 0], v[:2, 1] = 1.0, 50.0  # the first of them starts nearer, off to the side
    v[512:520] = np.repeat([[5.0, 0.0, 0.0, 0.0], [5.1, 0.0, 0.0, 0.0], [5.2, 0.0, 0.0, 0.0], [5.3, 0.0, 0.0, 0.0]], 2, 0)
    v[513:520:2, 0] += 0.2
    v[520:, :3] = [[far, far, far], [far, -far, -far]]  # the scene as wide as it is long: the first one in their cell
    v[:, 3] = 1.0
    rays = np.zeros((many, 8))
    rays[:, 1:3] = rng.uniform(-0.05, 0.05, (many, 2))
    rays[:, 4] = 1.0
    rays[:, 7] = np.inf
    v, rays[:, :3], rays[:, 4:7] = v * scale, rays[:, :3] * scale, rays[:, 4:7] * scale
    idx = np.arange(522, dtype=np.int32).reshape(261, 2)
    vt, it = torch.from_numpy(v.astype(np.float32)).cuda(), torch.from_numpy(idx).cuda()
    r = torch.from_numpy(rays.astype(np.float32)).cuda()
    b = api.lbvh_build_boxes(api.lss_bounds(vt, it))
    u = torch.zeros(many, device="cuda"), torch.zeros(few, device="cuda")
    full, part = api.trace_lss(b, vt, it, r, u=u[0]), api.trace_lss(b, vt, it, r[:few].contiguous(), u=u[1])
    assert int(torch.isnan(full[:few, 1].view(torch.float32)).sum()) > few // 2
    assert torch.equal(full[:few], part)
    assert torch.equal(u[0][:few].view(torch.int32), u[1].view(torch.int32))
