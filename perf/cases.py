"""The work that programs have this library do, as measurable cases.

Seven families, each through the package's public calls with the plans, work
space and output buffers that a program keeps between calls:

  scan       prefix sums, partition and select (api.exclusive_sum, ...)
  sort       stable radix sorts of keys with payloads (api.sort)
  mesh       one triangle mesh: build or refit, then trace the binary LBVH
  wide       one mesh per frame: build, collapse to the 8-wide quantised BVH,
             closest hits of the primary rays, occlusion of a second ray set
  batch      many meshes in one build, collapse and trace
  prims      spheres or swept spheres: bounds, box LBVH, trace
  solids     point location in a volume mesh of linear cells
  instances  instanced meshes: top-level rebuild, trace

Sizes are those of the benchmark and the tests (bench.py, workloads.py,
tests/cpp) and generic odd ones between them.
"""
import numpy as np
import torch

from gprt_b200 import api, lib, scenes

INT_MAX = 2 ** 31 - 1


def listed():
    return [
        # The smallest call: the last size of the scan test's schedule
        # (multiples of 9973), where the launch is the cost.
        {"name": "scan_small", "family": "scan", "op": "exclusive", "n": 99_730},
        # Stream compaction of a large signed array (the benchmark's uniform
        # int32 values at about 2^30), an odd count.
        {"name": "partition_large", "family": "scan", "op": "partition", "n": 1_000_000_007},
        # The small plain configuration: 2^20 uniform pairs.
        {"name": "sort_small", "family": "sort", "key": 4, "value": 4, "n": 1 << 20, "keys": "uniform"},
        # The benchmark's sort: 2^28 Zipf(1.1) pairs.
        {"name": "sort_large", "family": "sort", "key": 4, "value": 4, "n": 1 << 28, "keys": "zipf"},
        # The reference's untyped form, 64-bit keys with 64-bit payloads, at
        # the count of its sort test.
        {"name": "sort_u64", "family": "sort", "key": 8, "value": 8, "n": 100_000_000, "keys": "uniform"},
        # A small object picked or sampled by few rays: latency of the whole
        # chain of a build and a trace.
        {"name": "mesh_small", "family": "mesh", "n": 1_501, "rays": 4_099, "code": 0, "refit": False, "any": False,
         "sigma": 0.05},
        # The small LBVH configuration.
        {"name": "mesh_plain", "family": "mesh", "n": 262_144, "rays": 1_048_576, "code": 0, "refit": False,
         "any": False, "sigma": 0.002},
        # An ordinary frame over the quantised BVH: rebuild, primary rays,
        # shadow rays; a quarter of the benchmark's wide scene, ragged.
        {"name": "wide_frame", "family": "wide", "n": 4_194_301, "rays": 4_000_037, "clusters": 64},
        # The batched configuration: 4,096 meshes of log-uniform size in
        # [64, 65536], two rays per triangle.
        {"name": "batch_large", "family": "batch", "meshes": 4_096, "most": 65_536, "rays_per_tri": 2},
        # Hair: swept spheres of 16-segment strands, the benchmark's count
        # divided by four.
        {"name": "lss", "family": "prims", "kind": "lss", "n": 1_048_576, "rays": 1_048_577, "exit": False},
        # Sampling a volume mesh: the benchmark's grid, a quarter of its points.
        {"name": "solids", "family": "solids", "g": 96, "points": 4_194_301},
        # The benchmark's instanced scene, a quarter of its rays.
        {"name": "instances", "family": "instances", "meshes": 64, "n": 4_194_304, "instances": 16_384,
         "rays": 4_194_304},
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], log-uniform, odd more often than not."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(lo, min(hi, v | 1 if rng.random() < 0.7 else v))


def draw(rng):
    family = rng.choice(("scan", "sort", "sort", "mesh", "mesh", "wide", "wide", "batch", "prims", "solids", "instances"))
    if family == "scan":
        return {"family": family, "op": rng.choice(("exclusive", "inclusive", "partition", "select")),
                "n": _log(rng, 9_973, 1_000_000_000)}
    if family == "sort":
        key, value = rng.choice(((4, 0), (4, 4), (4, 8), (8, 0), (8, 4), (8, 8)))
        return {"family": family, "key": key, "value": value,
                "n": _log(rng, 20_000, 200_000_000 if key + value <= 8 else 80_000_000),
                "keys": rng.choice(("uniform", "zipf"))}
    if family == "mesh":
        n = _log(rng, 500, 1_000_000)
        return {"family": family, "n": n, "rays": _log(rng, 2_000, 2_000_000), "code": rng.choice((0, 0, 1)),
                "refit": rng.random() < 0.3, "any": rng.random() < 0.3, "sigma": 0.1 / n ** (1.0 / 3.0)}
    if family == "wide":
        return {"family": family, "n": _log(rng, 20_000, 4_194_301), "rays": _log(rng, 20_000, 4_000_000),
                "clusters": rng.choice((16, 64, 256))}
    if family == "batch":
        return {"family": family, "meshes": _log(rng, 16, 4_096), "most": _log(rng, 128, 65_536),
                "rays_per_tri": rng.choice((1, 2))}
    if family == "prims":
        return {"family": family, "kind": rng.choice(("spheres", "lss")), "n": _log(rng, 10_000, 1_048_576),
                "rays": _log(rng, 10_000, 1_048_577), "exit": rng.random() < 0.2}
    if family == "solids":
        return {"family": family, "g": _log(rng, 12, 96), "points": _log(rng, 20_000, 4_194_301)}
    return {"family": family, "meshes": rng.choice((1, 4, 16, 64)), "n": _log(rng, 50_000, 4_194_304),
            "instances": _log(rng, 64, 16_384), "rays": _log(rng, 20_000, 4_194_304)}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _off32(off):
    return torch.from_numpy(np.asarray(off, np.int64).astype(np.uint32).view(np.int32)).cuda()


def _mesh_sizes(c):
    """Triangles of each mesh of a batch: log-uniform in [64, most], the same
    for every seed."""
    r = np.random.default_rng(2024 + c["meshes"])
    return np.floor(np.exp(r.uniform(np.log(64), np.log(c["most"]), size=c["meshes"]))).astype(np.int64)


def _sort_inputs(c, seed):
    g, n, kw, vw = _gen(seed, 1), c["n"], c["key"], c["value"]
    kt = torch.int32 if kw == 4 else torch.int64
    if c["keys"] == "zipf":  # Zipf(1.1) by inversion, as the benchmark draws it
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        keys = ((1.0 - u) ** -10.0).floor_().clamp_(1, 2 ** 32 - 1).sub_(1).to(torch.int64).to(kt)
    elif kw == 4:
        keys = torch.randint(-INT_MAX - 1, INT_MAX + 1, (n,), generator=g, device="cuda", dtype=kt)
    else:
        keys = torch.randint(-2 ** 63, 2 ** 63 - 1, (n,), generator=g, device="cuda", dtype=kt)
    vals = torch.arange(n, device="cuda", dtype=torch.int32 if vw == 4 else torch.int64) if vw else None
    return keys, vals


def _scan_input(c, seed):
    g = _gen(seed, 2)
    if c["op"] in ("partition", "select"):
        return torch.randint(-INT_MAX - 1, INT_MAX + 1, (c["n"],), generator=g, device="cuda", dtype=torch.int32)
    return torch.randint(0, 256, (c["n"],), generator=g, device="cuda", dtype=torch.int32)


def _mesh_inputs(c, seed):
    pos, tri = api.gen_soup(c["n"], seed=2 * seed + 11, sigma=c["sigma"])
    return pos, tri, api.gen_rays(c["rays"], seed=2 * seed + 12)


def _lss_strands(n, g):
    """Hair: random walks of 16 segments, the radius tapering to half."""
    segs, strands = 16, -(-n // 16)
    start = torch.rand((strands, 1, 3), generator=g, device="cuda")
    steps = torch.randn((strands, segs, 3), generator=g, device="cuda") * 0.004
    p = torch.cat([start, start + torch.cumsum(steps, 1)], 1)
    r = 0.0005 + 0.001 * torch.rand((strands, 1), generator=g, device="cuda")
    r = r * (1.0 - 0.5 * torch.arange(segs + 1, device="cuda") / segs)
    verts = torch.cat([p, r[:, :, None]], 2).reshape(-1, 4).contiguous()
    first = (torch.arange(strands, device="cuda") * (segs + 1))[:, None] + torch.arange(segs, device="cuda")
    idx = torch.stack([first, first + 1], 2).reshape(-1, 2)[:n].to(torch.int32).contiguous()
    return verts, idx


def _instance_records(c, seed):
    """Placements: random rotation, scale in [0.5, 2], translation in
    [0, 24]^3, the masks cycling through four bits."""
    r = np.random.default_rng(seed)
    rec = np.zeros(c["instances"], np.dtype(api.INSTANCE_DTYPE))
    q, _ = np.linalg.qr(r.normal(size=(c["instances"], 3, 3)))
    m = np.zeros((c["instances"], 3, 4))
    m[:, :, :3] = q * r.uniform(0.5, 2.0, (c["instances"], 1, 1))
    m[:, :, 3] = r.uniform(0.0, 24.0, (c["instances"], 3))
    i = np.arange(c["instances"])
    rec["transform"] = m.reshape(-1, 12)
    rec["custom_mask"] = ((1 << (i % 4)) << 24) | i
    rec["blas"] = i % c["meshes"]
    return rec


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    c = dict(case)
    s = {"case": c}
    fam = c["family"]
    if fam == "scan":
        s["in"] = _scan_input(c, seed)
        s["out"] = torch.zeros_like(s["in"])
        s["total"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        s["scr"] = api.scratch(api.scan_scratch_size(c["n"]))
        return s
    if fam == "sort":
        s["keys"], s["vals"] = _sort_inputs(c, seed)
        s["k"] = torch.empty_like(s["keys"])
        s["v"] = None if s["vals"] is None else torch.empty_like(s["vals"])
        s["scr"] = api.scratch(api.sort_scratch_size(c["n"], c["key"], c["value"]))
        return s
    s["tscr"] = api.scratch(lib().gprtcuTraceScratchSize())
    if fam == "mesh":
        s["pos"], s["tri"], s["rays"] = _mesh_inputs(c, seed)
        s["bvh"] = api.Lbvh(c["n"])
        if c["refit"]:  # built once; the vertices have moved since
            api.lbvh_build_triangles(s["pos"], s["tri"], s["bvh"], code_kind=c["code"])
            move = torch.randn((c["n"], 1, 3), generator=_gen(seed, 3), device="cuda") * c["sigma"]
            s["pos"] = (s["pos"].view(c["n"], 3, 3) + move).reshape(-1, 3).contiguous()
    elif fam == "wide":
        s["pos"], s["tri"] = api.gen_mixture(c["n"], clusters=c["clusters"], seed=2 * seed + 3)
        s["rays"] = api.gen_rays(c["rays"], seed=2 * seed + 4)
        s["shadow"] = api.gen_rays(c["rays"], seed=2 * seed + 100_005)
        s["bvh"] = api.Lbvh(c["n"], with_aabbs=False)
        s["wide"] = api.WideBvh(c["n"])
        s["hits2"] = torch.empty((c["rays"], 2), dtype=torch.int32, device="cuda")
    elif fam == "batch":
        sizes = _mesh_sizes(c)
        off = np.zeros(sizes.size + 1, np.int64)
        off[1:] = np.cumsum(sizes)
        n = int(off[-1])
        s["pos"], s["tri"] = api.gen_mixture(n, clusters=256, seed=2 * seed + 5)
        s["batch"] = api.BatchLbvh(off, with_aabbs=False)
        s["wide"] = api.WideBvh(n, sizes.size)
        s["ray_off"] = _off32(off * c["rays_per_tri"])
        tri_box = s["pos"].view(n, 3, 3)
        m = torch.repeat_interleave(torch.arange(sizes.size, device="cuda"), torch.from_numpy(sizes).cuda())
        m = m[:, None].expand(n, 3)
        box = torch.empty((sizes.size, 6), device="cuda")
        box[:, :3] = torch.full((sizes.size, 3), 1e30, device="cuda").scatter_reduce_(0, m, tri_box.amin(1), "amin")
        box[:, 3:] = torch.full((sizes.size, 3), -1e30, device="cuda").scatter_reduce_(0, m, tri_box.amax(1), "amax")
        c["rays"] = n * c["rays_per_tri"]
        s["rays"] = api.gen_rays(c["rays"], seed=2 * seed + 6, ray_off=s["ray_off"], meshes=sizes.size, boxes=box)
    elif fam == "prims":
        g = _gen(seed, 4)
        if c["kind"] == "spheres":
            s["prims"] = torch.rand((c["n"], 4), generator=g, device="cuda")
            s["prims"][:, 3].mul_(0.0015).add_(0.0005)
        else:
            s["prims"], s["idx"] = _lss_strands(c["n"], g)
        s["rays"] = api.gen_rays(c["rays"], seed=2 * seed + 8)
        s["boxes"] = torch.empty((c["n"], 6), device="cuda")
        s["bvh"] = api.Lbvh(c["n"])
        s["u"] = torch.empty(c["rays"], device="cuda")
    elif fam == "solids":
        # every fill of a cube equally often, so each seed has as many cells
        fills = np.random.default_rng(seed).permutation(np.resize(np.arange(len(scenes.SOLID_FILLS)), c["g"] ** 3))
        verts, idx, types = scenes.solid_grid(c["g"], seed=seed, fills=fills)
        n = types.size
        s["solids"] = api.Solids(torch.from_numpy(verts).cuda(), torch.from_numpy(idx.view(np.int32)).cuda(),
                                 torch.from_numpy(types).cuda())
        s["points"] = torch.rand((c["points"], 4), generator=_gen(seed, 5), device="cuda")
        s["aabbs"] = torch.empty((n, 8), device="cuda")
        s["boxes"] = torch.empty((n, 6), device="cuda")
        s["bvh"] = api.Lbvh(n)
        s["hits"] = torch.empty((c["points"], 2), dtype=torch.int32, device="cuda")
        s["rstw"] = torch.empty((c["points"], 4), device="cuda")
        return s
    else:
        off = np.linspace(0, c["n"], c["meshes"] + 1).astype(np.int64)
        s["pos"], s["tri"] = api.gen_mixture(c["n"], clusters=c["meshes"], seed=2 * seed + 11, edge_sigma=0.002)
        if c["meshes"] > 1:
            s["blas"] = api.BatchLbvh(off, with_aabbs=False)
            api.batch_build_triangles(s["pos"], s["tri"], s["blas"])
        else:
            s["blas"] = api.Lbvh(c["n"], with_aabbs=False)
            api.lbvh_build_triangles(s["pos"], s["tri"], s["blas"])
        s["tlas"] = api.Tlas(api.instances_tensor(_instance_records(c, seed)), s["blas"].root, c["meshes"])
        world = torch.tensor([-1.0, -1.0, -1.0, 25.0, 25.0, 25.0], device="cuda")
        s["rays"] = api.gen_rays(c["rays"], seed=2 * seed + 12, boxes=world)
        s["inst"] = torch.empty(c["rays"], dtype=torch.int32, device="cuda")
    s["hits"] = torch.empty((c["rays"], 2), dtype=torch.int32, device="cuda")
    return s


def _hits(h):
    """A hit record's two words: the primitive and its distance."""
    return {"prim": h[:, 0], "t": h[:, 1].view(torch.float32)}


# --------------------------------------------------------------------- run
def run(s):
    c = s["case"]
    fam = c["family"]
    if fam == "scan":
        if c["op"] in ("exclusive", "inclusive"):
            f = api.exclusive_sum if c["op"] == "exclusive" else api.inclusive_sum
            out, total = f(s["in"], out=s["out"], total=s["total"], scr=s["scr"])
        else:
            f = api.partition if c["op"] == "partition" else api.select
            out, total = f(s["in"], out=s["out"], count=s["total"], scr=s["scr"])
        return {"out": out, "total": total}
    if fam == "sort":
        # the sort is in place, and the program still needs its unsorted data
        s["k"].copy_(s["keys"])
        if s["vals"] is not None:
            s["v"].copy_(s["vals"])
        keys, vals = api.sort(s["k"], s["v"], scr=s["scr"])
        return {"keys": keys, "values": vals}
    if fam == "mesh":
        b = s["bvh"]
        if c["refit"]:
            api.lbvh_refit_triangles(s["pos"], s["tri"], b)
        else:
            api.lbvh_build_triangles(s["pos"], s["tri"], b, code_kind=c["code"])
        h = api.trace(b, s["rays"], hits=s["hits"], anyhit=c["any"], scr=s["tscr"])
        return {"codes": b.codes, "ids": b.ids, "nodes": b.nodes, "aabbs": b.aabbs, "root": b.root, **_hits(h)}
    if fam == "wide":
        api.lbvh_build_triangles(s["pos"], s["tri"], s["bvh"])
        api.wide_build(s["bvh"], wide=s["wide"])
        h = api.wide_trace(s["wide"], s["rays"], hits=s["hits"], scr=s["tscr"])
        d = api.wide_trace(s["wide"], s["shadow"], hits=s["hits2"], anyhit=True, scr=s["tscr"])
        # a shadow ray asks whether something is in the way; which of the
        # triangles in the way is reported is left open by the call
        return {**_hits(h), "occluded": d[:, 0].ne(-1)}
    if fam == "batch":
        api.batch_build_triangles(s["pos"], s["tri"], s["batch"])
        api.wide_build(s["batch"], wide=s["wide"])
        return _hits(api.wide_trace(s["wide"], s["rays"], s["ray_off"], hits=s["hits"], scr=s["tscr"]))
    if fam == "prims":
        if c["kind"] == "spheres":
            api.sphere_bounds(s["prims"], out=s["boxes"])
            api.lbvh_build_boxes(s["boxes"], s["bvh"])
            h = api.trace_spheres(s["bvh"], s["prims"], s["rays"], s["hits"], s["u"], exit_test=c["exit"],
                                  scr=s["tscr"])
        else:
            api.lss_bounds(s["prims"], s["idx"], out=s["boxes"])
            api.lbvh_build_boxes(s["boxes"], s["bvh"])
            h = api.trace_lss(s["bvh"], s["prims"], s["idx"], s["rays"], hits=s["hits"], u=s["u"],
                              exit_test=c["exit"], scr=s["tscr"])
        return {"boxes": s["boxes"], "u": s["u"], **_hits(h)}
    if fam == "solids":
        api.solid_bounds(s["solids"], s["aabbs"], s["boxes"])
        api.lbvh_build_boxes(s["boxes"], s["bvh"])
        hits, rstw = api.locate_solid_points(s["bvh"], s["solids"], s["points"], s["hits"], s["rstw"], scr=s["tscr"])
        return {"boxes": s["boxes"], "aabbs": s["aabbs"], "cell": hits, "rstw": rstw}
    s["tlas"].build()
    off = s["blas"].tri_off if c["meshes"] > 1 else None
    h, inst = api.trace_instances(s["tlas"], s["blas"], s["rays"], off, c["meshes"], 0xFF, s["hits"], s["inst"],
                                  scr=s["tscr"])
    return {"instance": inst, **_hits(h)}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes that one pass cannot do without: every input read once and every
    documented output written once.  Arithmetic is counted only where the
    number of tests does not depend on the traversal, so it is left at zero."""
    c, fam = case, case["family"]
    if fam == "scan":
        b = c["n"] * (6 if c["op"] == "select" else 8)
    elif fam == "sort":
        b = 2 * c["n"] * (c["key"] + c["value"])
    elif fam == "mesh":
        # indices and vertices in; codes, ids, nodes, boxes out; rays, hits
        b = c["n"] * (48 + (48 if c["refit"] else 88)) + c["rays"] * 40
    elif fam == "wide":
        b = c["n"] * (48 + 40) + 2 * c["rays"] * 40
    elif fam == "batch":
        n = int(_mesh_sizes(c).sum())
        b = n * (48 + 40 + 40 * c["rays_per_tri"])
    elif fam == "prims":
        b = c["n"] * (16 + (8 if c["kind"] == "lss" else 0) + 24 + 88) + c["rays"] * 44
    elif fam == "solids":
        # 3.2 cells and two vertices per cube on average
        b = int(c["g"] ** 3 * (3.2 * (33 + 56 + 88) + 32)) + c["points"] * (16 + 8 + 16)
    else:
        b = c["instances"] * (64 + 72 + 88) + c["n"] * 48 + c["rays"] * 44
    return {"bytes": b, "flops": 0}


# ------------------------------------------------------------------- exact
def _exact_small_mesh(c, seed):
    """Closest hit of every ray by testing every triangle in 64 bits (plane
    distance and signed edge volumes); inf where there is none."""
    pos, tri, rays = _mesh_inputs(c, seed)
    v = pos[tri.long()].double()  # [n, 3, 3]
    out = []
    for r in rays.double().split(256):
        o, d = r[:, None, :3], r[:, None, 4:7]
        a, b, e = (v[None, :, k] - o for k in range(3))
        dd = d.expand_as(a)
        u = (torch.linalg.cross(e, b) * dd).sum(-1)
        w = (torch.linalg.cross(a, e) * dd).sum(-1)
        x = (torch.linalg.cross(b, a) * dd).sum(-1)
        inside = ((u >= 0) & (w >= 0) & (x >= 0)) | ((u <= 0) & (w <= 0) & (x <= 0))
        nrm = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])[None]
        den = (nrm * dd).sum(-1)
        t = (nrm * a).sum(-1) / den
        ok = inside & (den != 0) & (t >= r[:, None, 3]) & (t <= r[:, None, 7])
        out.append(torch.where(ok, t, torch.inf).amin(1))
    return torch.cat(out)


def exact(case, seed):
    c, fam = case, case["family"]
    if fam == "scan":
        x = _scan_input(c, seed).long()
        if c["op"] in ("exclusive", "inclusive"):
            inc = x.cumsum(0)
            total = inc[-1:].clone()
            return {"out": inc if c["op"] == "inclusive" else inc.sub_(x), "total": total}
        sel = x[x >= 0]
        rest = x[x < 0].flip(0) if c["op"] == "partition" else x.new_zeros(x.numel() - sel.numel())
        return {"out": torch.cat([sel, rest]), "total": torch.tensor([sel.numel()])}
    if fam == "sort":
        # unsigned order: flip the sign bit, sort as signed, flip it back
        keys, vals = _sort_inputs(c, seed)
        k = keys.long() & 0xFFFFFFFF if c["key"] == 4 else keys ^ (-2 ** 63)
        k, at = torch.sort(k, stable=True)
        return {"keys": k if c["key"] == 4 else k ^ (-2 ** 63), "values": None if vals is None else vals[at]}
    if fam == "mesh" and not c["any"] and not c["refit"] and c["n"] * c["rays"] <= 40_000_000:
        # the distance; the arrays of the build are whole numbers and minima
        # and maxima of the input
        return {k: None for k in ("codes", "ids", "nodes", "aabbs", "root", "prim")} | {"t": _exact_small_mesh(c, seed)}
    # Testing every primitive against every ray would take minutes, and the
    # cells' and swept spheres' answers hang on the iteration and the cut-offs
    # that the 32-bit call documents.
    return None
