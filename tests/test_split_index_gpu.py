"""The position-staged split (from 8, 16 or 32 buckets on, by layout) at tile
edges, in both of its rankings: the quick one with its check, and the exact one
that a tile takes when the check fails; skewed keys, every key in one bucket,
one launch and three launches."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

LAYOUTS = {"ko": 0, "aos": 1, "soa": 2}


def _want(torch, keys, vals, buckets):
    b = (keys & (buckets - 1)).long()
    order = torch.sort(b, stable=True)[1]
    counts = torch.bincount(b, minlength=buckets)
    return keys[order], vals[order], (torch.cumsum(counts, 0) - counts).to(torch.int32)


def _split(edpp, torch, keys, vals, buckets, layout, exact):
    n = keys.numel()
    src = torch.stack([keys, vals], 1).contiguous() if layout == "aos" else keys
    out = torch.full_like(src, -1)
    vo = torch.full_like(vals, -1)
    start = torch.empty(buckets, dtype=torch.int32, device="cuda")
    ws = edpp.workspace(edpp.split_workspace_bytes(n, buckets, layout))
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    soa = layout == "soa"
    f = edpp.lib().edpp_selftest_split_exact if exact else edpp.lib().edpp_split_i32
    edpp.check(f(p(src), p(out), p(start), n, buckets, LAYOUTS[layout], p(vals) if soa else None,
                 p(vo) if soa else None, p(ws), ws.numel(), edpp.current_stream_handle()))
    if layout == "aos":
        return out[:, 0], out[:, 1], start
    return out, (vo if soa else None), start


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("layout", ["ko", "soa", "aos"])
@pytest.mark.parametrize("buckets", [8, 16, 32, 64, 128, 256, 512, 1024])
def test_both_rankings(cuda, edpp, buckets, layout, exact):
    g = cuda.Generator(device="cuda")
    # one launch up to 2.4 million elements, three launches above
    for n in (1, 33, 6143, 6145, 8191, 8193, 100_003, (1 << 22) + 8192, 6144 * 700, 6144 * 700 + 1):
        g.manual_seed(n + buckets)
        vals = cuda.arange(n, device="cuda", dtype=cuda.int32)
        uniform = cuda.randint(-2**31, 2**31 - 1, (n,), generator=g, device="cuda", dtype=cuda.int32)
        one = uniform & ~(buckets - 1) | (buckets - 1)
        skew = cuda.where(uniform > 0, one, uniform)
        ordered = cuda.sort(uniform & (buckets - 1))[0]
        ends = uniform.clone()  # a warp's first and last element share a bucket
        ends[::128] = 5
        ends[127::128] = 5
        for keys in (uniform, one, skew, ordered, ends):
            wk, wv, ws = _want(cuda, keys, vals, buckets)
            k, v, s = _split(edpp, cuda, keys, vals, buckets, layout, exact)
            assert cuda.equal(k, wk) and cuda.equal(s, ws), n
            assert v is None or cuda.equal(v, wv), n
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("layout,buckets", [("ko", 2), ("ko", 1024), ("soa", 64), ("soa", 256),
                                            ("aos", 256)])
def test_four_tiles_per_histogram_block(cuda, edpp, layout, buckets):
    # from 4864 tiles on a histogram block counts four; rows padded to four tiles
    tile = 6144 if layout != "ko" and buckets <= 64 else 8192
    for n in (4864 * tile - tile, 4864 * tile, 4864 * tile + 1, 4866 * tile - 3):
        vals = cuda.arange(n, device="cuda", dtype=cuda.int32)
        keys = cuda.randint(-2**31, 2**31 - 1, (n,), device="cuda", dtype=cuda.int32)
        wk, wv, ws = _want(cuda, keys, vals, buckets)
        k, v, s = _split(edpp, cuda, keys, vals, buckets, layout, False)
        assert cuda.equal(k, wk) and cuda.equal(s, ws), n
        assert v is None or cuda.equal(v, wv), n
