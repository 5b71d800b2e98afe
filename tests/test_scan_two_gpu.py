"""The two-launch scan of middle sizes (256 KB to 48 MB, 64-bit 32 MB) at the
edges of its range, of its tiles (32 KB) and of the strides in which the tile
sums are added up; unaligned and in place; infinities and NaN; captured in a
CUDA graph; on two streams at once."""
import pytest

pytestmark = pytest.mark.gpu

TILE_BYTES, SMALL_BYTES = 32768, 256 << 10


def _lengths(elem):
    small, top = SMALL_BYTES // elem, ((48 if elem == 4 else 32) << 20) // elem
    tile = TILE_BYTES // elem
    return [small + 1, small + tile - 1, small + tile, small + tile + 1, 256 * tile, 257 * tile + 3,
            513 * tile - 1, top - 1, top, top + 1]


@pytest.fixture(autouse=True)
def default_table(edpp):
    edpp.tune_load(None)


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("dt", ["int32", "int64"])
def test_edges(cuda, edpp, dt, algo):
    tdt = getattr(cuda, dt)
    lim = 2**31 if dt == "int32" else 2**62
    for n in _lengths(4 if dt == "int32" else 8):
        buf = cuda.randint(-lim, lim - 1, (n + 1,), dtype=tdt, device="cuda")
        for off in (0, 1):  # one element in: off 16-byte alignment
            x = buf[off:off + n]
            ref = cuda.cumsum(x.to(cuda.int64), 0).to(tdt)  # wraps
            y = cuda.empty(n + 1, dtype=tdt, device="cuda")[off:off + n]
            assert cuda.equal(edpp.scan(x, algo=algo, out=y), ref - x), (n, off)
            assert cuda.equal(edpp.scan(x, inclusive=True, algo=algo, out=x), ref), (n, off)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("algo", ["lookback", "rts"])
def test_f32_error_and_special_values(cuda, edpp, algo):
    for n in _lengths(4):
        x = cuda.rand(n, device="cuda") * 2 - 1
        ref = cuda.cumsum(x.double(), 0)
        y = edpp.scan(x, inclusive=True, algo=algo)
        # in its tile a sum passes through at most 3 + 5 + 2 + 5 + 2 additions of
        # values within the tile's sum of |x|, and through three roundings with
        # the prefix: 24 roundings of 2^-24; a tile's sum leaves out two per
        # chunk of four, at random, so at most 2 * 2^-24 * 4 * 6 * sqrt(chunks)
        u = 2.0**-24
        lim = u * (24 * (ref.abs().max().item() + TILE_BYTES / 4) + 48 * (n / 4)**0.5)
        assert (y.double() - ref).abs().max().item() <= lim, n
        assert cuda.equal(edpp.scan(x, inclusive=True, algo=algo), y)  # the same bits
    n = 1_000_003
    for at, v in ((0, float("inf")), (500_000, float("-inf")), (700_000, float("nan")),
                  (300_000, 3e38)):
        z = cuda.rand(n, device="cuda")
        z[at:at + 2] = v
        y = edpp.scan(z, inclusive=True, algo=algo)
        ref = cuda.cumsum(z.double(), 0).float()
        assert cuda.equal(cuda.isnan(y), cuda.isnan(ref)) and cuda.equal(cuda.isinf(y), cuda.isinf(ref))
        assert cuda.equal(y[:at].isfinite(), cuda.ones_like(y[:at], dtype=cuda.bool))


def test_captured_and_on_two_streams(cuda, edpp):
    n = 3_000_017
    x = cuda.randint(-9, 9, (n,), dtype=cuda.int32, device="cuda")
    need = edpp.scan_workspace_bytes(n, "int32")
    y, ws = cuda.zeros_like(x), edpp.workspace(need)
    edpp.scan(x, inclusive=True, out=y, ws=ws)
    cuda.cuda.synchronize()
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):  # the second scan's sums come after the first's last read
        edpp.scan(x, inclusive=True, out=y, ws=ws)
        edpp.scan(y, inclusive=True, out=y, ws=ws)
    ref = cuda.cumsum(cuda.cumsum(x.long(), 0), 0).to(cuda.int32)
    for _ in range(3):
        y.zero_()
        g.replay()
        assert cuda.equal(y, ref)
    ref = cuda.cumsum(x, 0).to(cuda.int32)
    outs = []
    streams = [cuda.cuda.Stream(), cuda.cuda.Stream()]
    cuda.cuda.synchronize()
    for k in range(16):
        with cuda.cuda.stream(streams[k % 2]):
            o, w = cuda.zeros_like(x), edpp.workspace(need)
            edpp.scan(x, inclusive=True, out=o, ws=w)
            outs.append((o, w))
    cuda.cuda.synchronize()
    assert all(cuda.equal(o, ref) for o, _ in outs)
    assert edpp.sync_status() == edpp.EDPP_OK
