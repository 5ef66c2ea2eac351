"""The sort's default routes by size: one CTA up to 8,192 keys, then tiles that
grow with n.  Sizes either side of every line, all key/payload types, bit
ranges that are not whole digits, skewed keys; against a stable host sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = [(4, 0), (4, 4), (4, 8), (8, 0), (8, 4), (8, 8)]


def _check(kw, vw, n, begin, end, skew, seed):
    import torch
    from gprt_b200 import api
    rng = np.random.default_rng(seed)
    kt, vt = (np.uint32, np.uint64)[kw == 8], (np.uint32, np.uint64)[vw == 8]
    k = rng.integers(0, 2 ** (8 * kw), size=n, dtype=np.uint64)
    if skew:
        k = np.where(rng.random(n) < 0.8, k & np.uint64(0x0F000F), k) | (np.uint64(3) << np.uint64(8 * kw - 4))
        k[::17] = 2 ** (8 * kw) - 1
    k = k.astype(kt)
    v = np.arange(n).astype(vt) if vw else None
    masked = (k.astype(np.uint64) >> np.uint64(begin)) & np.uint64((1 << (end - begin)) - 1)
    at = np.argsort(masked, kind="stable")
    dk = torch.from_numpy(k.view(np.int32 if kw == 4 else np.int64)).cuda()
    dv = torch.from_numpy(v.view(np.int32 if vw == 4 else np.int64)).cuda() if vw else None
    scr = api.scratch(api.sort_scratch_size(n, kw, vw)).fill_(0xA5)
    api.sort(dk, dv, begin_bit=begin, end_bit=end, scr=scr)
    assert api.scratch_status(scr) == 0
    assert np.array_equal(dk.cpu().numpy().view(kt), k[at])
    if vw:
        assert np.array_equal(dv.cpu().numpy().view(vt), v[at])


@pytest.mark.parametrize("kw,vw", TYPES)
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1024, 1025, 1501, 4097, 8191, 8192, 8193])
def test_few_keys(cuda, kw, vw, n):
    for begin, end, skew in ((0, 8 * kw, False), (0, 30, True), (5, 18, False), (3, 4, True)):
        _check(kw, vw, n, begin, end, skew, n + begin)


@pytest.mark.parametrize("kw,vw", TYPES)
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 20) - 1, 1 << 20, 148 * 8192, 148 * 8192 + 1, 296 * 8192,
                               296 * 8192 + 1, (1 << 23) + 5])
def test_default_shapes(cuda, kw, vw, n):
    _check(kw, vw, n, 0, 8 * kw if n < (1 << 21) else 30, n % 2 == 0, n)


@pytest.mark.parametrize("n", [100, 8193, 20_001, 700_003])
@pytest.mark.parametrize("key,value", [(4, 4), (4, 8), (8, 4), (8, 8)])
@pytest.mark.parametrize("shift_k,shift_v", [(0, 1), (1, 0), (1, 1)])
def test_buffers_off_16_byte_boundaries(cuda, n, key, value, shift_k, shift_v):
    """Keys or payloads one element past an allocation's start: bulk copies
    cannot take them."""
    import torch
    from gprt_b200 import api
    k = np.random.default_rng(n).integers(0, 2 ** 12, n, dtype=np.uint64).astype(np.uint32 if key == 4 else np.uint64)
    kd = torch.zeros(n + 1, dtype=torch.int32 if key == 4 else torch.int64, device="cuda")[shift_k:shift_k + n]
    vd = torch.zeros(n + 1, dtype=torch.int32 if value == 4 else torch.int64, device="cuda")[shift_v:shift_v + n]
    kd.copy_(torch.from_numpy(k.view(np.int32 if key == 4 else np.int64)))
    vd.copy_(torch.arange(n))
    assert kd.data_ptr() % 16 == key * shift_k and vd.data_ptr() % 16 == value * shift_v
    api.sort(kd, vd)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(kd.cpu().numpy().view(k.dtype), k[order])
    assert np.array_equal(vd.cpu().numpy().astype(np.int64), order)


@pytest.mark.parametrize("key,value", TYPES)
def test_last_tile_lengths(cuda, key, value):
    """A last tile of every length modulo the 16 bytes that bulk copies move,
    from one key up, at each tile size of the default shapes."""
    import torch
    from gprt_b200 import api
    for tile in (1024, 2048, 4096, 6144, 8192):
        for rest in (1, 2, 3, 4, 5, 7, 15, tile // 2 + 1, tile - 3, tile - 1, tile):
            n = 3 * tile + rest
            k = np.random.default_rng(rest).integers(0, 2 ** 16, n, dtype=np.uint64).astype(
                np.uint32 if key == 4 else np.uint64)
            k[-1] = np.iinfo(k.dtype).max  # as large as what fills the tile up
            kd = torch.from_numpy(k.view(np.int32 if key == 4 else np.int64).copy()).cuda()
            vd = None if not value else torch.arange(n, device="cuda", dtype=torch.int32 if value == 4 else torch.int64)
            api.sort_with_config(kd, vd, (8, tile, 8))
            order = np.argsort(k, kind="stable")
            assert np.array_equal(kd.cpu().numpy().view(k.dtype), k[order]), n
            if value:
                assert np.array_equal(vd.cpu().numpy().astype(np.int64), order), n
