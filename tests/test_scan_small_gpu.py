"""Sums, partition and select of few tiles (one thread-block cluster) and just
past them: every tile count of the cluster, ragged ends, misaligned and aliased
buffers, scratch that holds garbage; against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 5, 8191, 8192, 8193, 3 * 8192, 4 * 8192 + 1, 8 * 8192, 8 * 8192 + 7, 99_730, 13 * 8192, 16 * 8192 - 3,
         16 * 8192, 16 * 8192 + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift", [0, 1])
def test_few_tile_sums(cuda, n, shift):
    import torch
    from gprt_b200 import api
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    inc = np.cumsum(x, dtype=np.uint64).astype(np.uint32)
    buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    d = buf[shift:shift + n]
    scr = api.scratch(api.scan_scratch_size(n)).fill_(0xA5)
    for inclusive in (False, True):
        for alias in (False, True):
            d.copy_(torch.from_numpy(x.view(np.int32)))
            out = d if alias else torch.empty_like(d)
            out, total = api.exclusive_sum(d, out=out, scr=scr, inclusive=inclusive)
            got = out.cpu().numpy().view(np.uint32)
            assert np.array_equal(got, inc if inclusive else inc - x)
            assert int(total.cpu().numpy().view(np.uint32)[0]) == int(inc[-1])
            assert api.scratch_status(scr) == 0


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("positive", [True, False])
def test_few_tile_partition(cuda, n, positive):
    import torch
    from gprt_b200 import api
    rng = np.random.default_rng(n + 1)
    x = rng.integers(-2 ** 31, 2 ** 31, size=n, dtype=np.int64).astype(np.int32)
    keep = (x >= 0) == positive
    for shift in (0, 1):
        buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
        d = buf[shift:shift + n]
        d.copy_(torch.from_numpy(x))
        scr = api.scratch(api.scan_scratch_size(n)).fill_(0xA5)
        out, count = api.partition(d, positive, scr=scr)
        assert int(count.item()) == int(keep.sum()) and api.scratch_status(scr) == 0
        assert np.array_equal(out.cpu().numpy(), np.concatenate([x[keep], x[~keep][::-1]]))
        out, count = api.select(d, positive, scr=scr)
        assert int(count.item()) == int(keep.sum())
        assert np.array_equal(out.cpu().numpy()[:int(keep.sum())], x[keep])
