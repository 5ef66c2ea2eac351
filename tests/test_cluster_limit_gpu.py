"""Calls that run as one thread-block cluster, on a device (here: with the
limit set by a test hook) where clusters of that size do not fit: the general
forms take them, with the same results."""
import numpy as np
import pytest

from gprt_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[1, 4, 8])
def limit(cuda, request):
    import gprt_b200
    gprt_b200.lib().gprtcuDebugMaxCluster(request.param)
    yield request.param
    gprt_b200.lib().gprtcuDebugMaxCluster(0)


@pytest.mark.parametrize("n", [5, 8193, 4 * 8192 + 1, 8 * 8192, 8 * 8192 + 7, 16 * 8192])
@pytest.mark.parametrize("shift", [0, 1])
def test_sums_and_partition(limit, n, shift):
    import torch
    from gprt_b200 import api
    x = np.random.default_rng(n).integers(-2 ** 31, 2 ** 31, size=n, dtype=np.int64).astype(np.int32)
    buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    d = buf[shift:shift + n]
    d.copy_(torch.from_numpy(x))
    scr = api.scratch(api.scan_scratch_size(n)).fill_(0xA5)
    inc = np.cumsum(x.view(np.uint32), dtype=np.uint64).astype(np.uint32)
    for inclusive in (False, True):
        out, total = api.exclusive_sum(d, scr=scr, inclusive=inclusive)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), inc if inclusive else inc - x.view(np.uint32))
        assert int(total.cpu().numpy().view(np.uint32)[0]) == int(inc[-1]) and api.scratch_status(scr) == 0
    out, count = api.partition(d, scr=scr)
    assert np.array_equal(out.cpu().numpy(), np.concatenate([x[x >= 0], x[x < 0][::-1]]))
    out, count = api.select(d, scr=scr)
    assert np.array_equal(out.cpu().numpy()[:int(count.item())], x[x >= 0]) and api.scratch_status(scr) == 0


@pytest.mark.parametrize("n", [1, 9, 700, 20000, 150001])
def test_collapse(limit, n):
    import torch
    from gprt_b200 import api
    pos, tri = scenes.soup(n, seed=n, sigma=0.02)
    b = api.lbvh_build_triangles(torch.from_numpy(pos).cuda(), torch.from_numpy(tri.view(np.int32)).cuda())
    rays = torch.from_numpy(scenes.rays(5000, seed=n)).cuda()
    w = api.wide_build(b)
    assert api.scratch_status(w.scratch) == 0
    assert torch.equal(api.wide_trace(w, rays), api.trace(b, rays))
