"""The default shape of a sort is close to the best of the ordinary ones where
a rule of its choice changes; the results are those of any shape."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _us(f):
    import torch
    f()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f()
    times = []
    for _ in range(9):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(20):
            graph.replay()
        e[1].record()
        e[1].synchronize()
        times.append(50 * e[0].elapsed_time(e[1]))
    return min(times[2:])


@pytest.mark.parametrize("key,value,n", [(4, 8, 700_001), (8, 4, 700_001), (8, 8, 700_001), (8, 8, 8_000_001),
                                         (8, 8, 9_000_001)])
def test_default_shape_time(cuda, key, value, n):
    import torch
    from gprt_b200 import api
    kt, vt = (torch.int32 if key == 4 else torch.int64), (torch.int32 if value == 4 else torch.int64)
    lim = 2 ** (8 * key - 1)
    g = torch.Generator("cuda").manual_seed(n)
    k0 = torch.randint(-lim, lim - 1, (n,), generator=g, device="cuda", dtype=kt)
    v0 = torch.arange(n, device="cuda", dtype=vt)
    k, v, scr = torch.empty_like(k0), torch.empty_like(v0), api.scratch(api.sort_scratch_size(n, key, value))

    def run(cfg):
        k.copy_(k0)
        v.copy_(v0)
        api.sort_with_config(k, v, cfg, scr=scr) if cfg else api.sort(k, v, scr=scr)

    others = {cfg: _us(lambda: run(cfg)) for cfg in ((8, 2048, 8), (8, 4096, 8), (8, 6144, 8), (8, 8192, 8))}
    ours = _us(lambda: run(None))
    assert ours < 1.05 * min(others.values()), (ours, others)


@pytest.mark.parametrize("key,value", [(4, 0), (4, 4), (4, 8), (8, 0), (8, 4), (8, 8)])
def test_sizes_around_the_lines(cuda, key, value):
    import torch
    from gprt_b200 import api
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (2 ** 19 - 1, 2 ** 19, sms * 4096, sms * 4096 + 1, sms * 6144, sms * 6144 + 1, sms * 8192, sms * 8192 + 1,
              7_499_999, 7_500_000, 11_500_000):
        if n > 2_000_000 and (key, value) != (8, 8):
            continue
        rng = np.random.default_rng(n)
        k = rng.integers(0, 2 ** (8 * key), n, dtype=np.uint64) >> np.uint64(8 * key - 20)  # many equal keys
        k = k.astype(np.uint32 if key == 4 else np.uint64)
        kd = torch.from_numpy(k.view(np.int32 if key == 4 else np.int64).copy()).cuda()
        vd = None if value == 0 else torch.arange(n, device="cuda", dtype=torch.int32 if value == 4 else torch.int64)
        api.sort(kd, vd)
        order = np.argsort(k, kind="stable")
        assert np.array_equal(kd.cpu().numpy().view(k.dtype), k[order])
        if value:
            assert np.array_equal(vd.cpu().numpy().astype(np.int64), order)


def test_ragged_last_tile_time(cuda):
    """A last tile that is nearly full costs what a full one does."""
    import torch
    from gprt_b200 import api
    times = []
    for n in (132 * 4096, 131 * 4096 + 3501):
        k0 = torch.randint(-2 ** 63, 2 ** 63 - 1, (n,), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
        v0 = torch.arange(n, device="cuda")
        k, v, scr = torch.empty_like(k0), torch.empty_like(v0), api.scratch(api.sort_scratch_size(n, 8, 8))

        def run():
            k.copy_(k0)
            v.copy_(v0)
            api.sort_with_config(k, v, (8, 4096, 8), scr=scr)

        times.append(_us(run))
    assert times[1] < 1.1 * times[0], times
