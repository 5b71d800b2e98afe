"""The one-launch split at the edges of its tile sizes (2048, 4096, 8192
elements), of the lengths that each takes (one, one and two tiles per SM) and
of the exchanged words (2^16); every layout, skewed keys, arrays off 16-byte
alignment, bucket starts, graph capture and two streams at once."""
import pytest

pytestmark = pytest.mark.gpu

WORDS = 1 << 16


def _want(torch, keys, vals, buckets):
    b = (keys & (buckets - 1)).long()
    order = torch.sort(b, stable=True)[1]
    counts = torch.bincount(b, minlength=buckets)
    return keys[order], vals[order], (torch.cumsum(counts, 0) - counts).to(torch.int32)


def _run(edpp, torch, keys, vals, buckets, layout):
    if layout == "aos":
        pairs = torch.stack([keys, vals], 1).contiguous()
        o, _, s = edpp.split(pairs, buckets, layout="aos", bucket_start=True)
        return o[:, 0], o[:, 1], s
    k, v, s = edpp.split(keys, buckets, values=vals if layout == "soa" else None, layout=layout,
                         bucket_start=True)
    return k, v, s


def _check(edpp, torch, n, buckets, layout, skew=False):
    g = torch.Generator(device="cuda")
    g.manual_seed(n * 31 + buckets)
    keys = torch.randint(-2**31, 2**31 - 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    if skew:
        keys = keys & ~(buckets - 1) | (buckets // 2)
        keys[::5] += 1 if buckets > 2 else 0
    vals = torch.arange(n, device="cuda", dtype=torch.int32)
    wk, wv, ws = _want(torch, keys, vals, buckets)
    k, v, s = _run(edpp, torch, keys, vals, buckets, layout)
    assert torch.equal(k, wk) and torch.equal(s, ws), (n, buckets, layout)
    assert v is None or torch.equal(v, wv), (n, buckets, layout)


@pytest.mark.parametrize("layout", ["ko", "soa", "aos"])
@pytest.mark.parametrize("buckets", [1, 2, 4, 16, 256, 1024])
def test_edges(cuda, edpp, buckets, layout):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    lengths = {1, 3, 2047, 2048, 2049}
    for tile, blocks in ((2048, sms), (4096, sms), (8192, 2 * sms)):
        last = tile * min(blocks, WORDS // buckets)  # the last length of this tile size
        lengths |= {last - 1, last, last + 1}
    for n in sorted(lengths):
        _check(edpp, cuda, n, buckets, layout)
        _check(edpp, cuda, n, buckets, layout, skew=True)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("buckets", [4, 64, 512])
def test_unaligned(cuda, edpp, buckets):
    n = 50_021
    keys = cuda.randint(0, 2**31 - 1, (n + 1,), device="cuda", dtype=cuda.int32)[1:]
    vals = cuda.arange(n + 3, device="cuda", dtype=cuda.int32)[3:]
    wk, wv, ws = _want(cuda, keys, vals, buckets)
    ko = cuda.empty(n + 2, device="cuda", dtype=cuda.int32)[2:]
    vo = cuda.empty(n + 1, device="cuda", dtype=cuda.int32)[1:]
    _, _, s = edpp.split(keys, buckets, values=vals, bucket_start=True, keys_out=ko, values_out=vo)
    assert cuda.equal(ko, wk) and cuda.equal(vo, wv) and cuda.equal(s, ws)


def test_captured_and_on_two_streams(cuda, edpp):
    n, buckets = 300_007, 64
    keys = cuda.randint(0, 2**31 - 1, (n,), device="cuda", dtype=cuda.int32)
    vals = cuda.arange(n, device="cuda", dtype=cuda.int32)
    wk, wv, _ = _want(cuda, keys, vals, buckets)
    need = edpp.split_workspace_bytes(n, buckets, "soa")
    ko, vo, ws = cuda.empty_like(keys), cuda.empty_like(vals), edpp.workspace(need)
    cuda.cuda.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        edpp.split(keys, buckets, values=vals, keys_out=ko, values_out=vo, ws=ws)
    for _ in range(3):
        ko.zero_()
        g.replay()
        assert cuda.equal(ko, wk) and cuda.equal(vo, wv)
    outs, streams = [], [cuda.cuda.Stream(), cuda.cuda.Stream()]
    cuda.cuda.synchronize()
    for k in range(8):
        with cuda.cuda.stream(streams[k % 2]):
            o = [cuda.empty_like(keys), cuda.empty_like(vals), edpp.workspace(need)]
            edpp.split(keys, buckets, values=vals, keys_out=o[0], values_out=o[1], ws=o[2])
            outs.append(o)
    cuda.cuda.synchronize()
    assert all(cuda.equal(o[0], wk) and cuda.equal(o[1], wv) for o in outs)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("n", [50_021, 3_000_001, 4864 * 8192 + 5])
def test_workspace_off_16_bytes(cuda, edpp, n):
    # a workspace 8 bytes past a 16-byte boundary: neither the one-launch form
    # nor the four-tile histogram reads or writes it in 16-byte words
    keys = cuda.randint(0, 2**31 - 1, (n,), device="cuda", dtype=cuda.int32)
    vals = cuda.arange(n, device="cuda", dtype=cuda.int32)
    wk, wv, s = _want(cuda, keys, vals, 256)
    ws = edpp.workspace(edpp.split_workspace_bytes(n, 256, "soa") + 8)[8:]
    k, v, st = edpp.split(keys, 256, values=vals, bucket_start=True, ws=ws)
    assert cuda.equal(k, wk) and cuda.equal(v, wv) and cuda.equal(st, s)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("layout", ["ko", "soa", "aos"])
@pytest.mark.parametrize("buckets", [1, 8, 16, 64, 256, 1024])
def test_counts_launch_edges(cuda, edpp, buckets, layout):
    # few words (2^13): the counts by a launch of their own, two tiles per SM at most
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    lengths = set()
    for tile in (2048, 4096, 8192):
        last = tile * min(2 * sms, (1 << 13) // buckets)
        lengths |= {last - 1, last, last + 1}
    for n in sorted(lengths):
        _check(edpp, cuda, n, buckets, layout)
        _check(edpp, cuda, n, buckets, layout, skew=True)
    assert edpp.sync_status() == edpp.EDPP_OK
