"""The pipelined one-launch scan (look-back variant 3, reduce-then-scan variant
0 for aligned arrays) at the edges of its tiles (16 KB), waves (one tile per SM)
and buffer ring (12 tiles per block); in place; captured in a CUDA graph; on
two streams at once; and the same f32 bits on every run."""
import pytest

pytestmark = pytest.mark.gpu

TILE_BYTES, STAGES = 16384, 12


@pytest.fixture
def pipe(edpp):
    edpp.lib().edpp_tune_clear()
    for elem in (4, 8):
        edpp.tune_set(edpp.TUNE_SCAN_LOOKBACK, elem, 20, 3)
        edpp.tune_set(edpp.TUNE_SCAN_RTS, elem, 20, 0)
    yield edpp
    edpp.tune_load(None)


def _lengths(torch, elem):
    tile = TILE_BYTES // elem
    wave = torch.cuda.get_device_properties(0).multi_processor_count * tile
    return [1, 3, tile - 1, tile, tile + 1, wave - 1, wave, wave + 1, wave + tile + 1,
            3 * wave - 5, STAGES * wave, (STAGES + 1) * wave + 2 * tile + 3,
            (2 * STAGES + 1) * wave + 7]


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("dt", ["int32", "int64"])
def test_edges(cuda, pipe, dt, algo):
    tdt = getattr(cuda, dt)
    lim = 2**31 if dt == "int32" else 2**62
    for n in _lengths(cuda, 4 if dt == "int32" else 8):
        x = cuda.randint(-lim, lim - 1, (n,), dtype=tdt, device="cuda")
        ref = cuda.cumsum(x.to(cuda.int64), 0).to(tdt)  # wraps
        assert cuda.equal(pipe.scan(x, inclusive=True, algo=algo), ref), n
        assert cuda.equal(pipe.scan(x, algo=algo), ref - x), n
        pipe.scan(x, inclusive=True, algo=algo, out=x)  # in place
        assert cuda.equal(x, ref), n
    assert pipe.sync_status() == pipe.EDPP_OK


def test_f32_error_and_repeatability(cuda, pipe):
    for n in _lengths(cuda, 4):
        x = cuda.rand(n, device="cuda") * 2 - 1
        ref = cuda.cumsum(x.double(), 0)
        y = pipe.scan(x, inclusive=True)
        # a sum passes through at most 4 + 5 + 5 + 5 additions in its tile, the
        # same in the reduction, 10 across the wave, and one rounding of the f64
        # carry: 40 roundings of 2^-24 of the largest partial sum of |x|
        lim = 40 * 2.0**-24 * (ref.abs().max().item() + TILE_BYTES / 4)
        assert (y.double() - ref).abs().max().item() <= lim, n
        assert cuda.equal(pipe.scan(x, inclusive=True), y)


def test_captured_and_on_two_streams(cuda, pipe):
    n = 5_000_003
    x = cuda.randint(-9, 9, (n,), dtype=cuda.int32, device="cuda")
    ref = cuda.cumsum(x, 0).to(cuda.int32)
    need = pipe.scan_workspace_bytes(n, "int32")
    y, ws = cuda.zeros_like(x), pipe.workspace(need)
    g = cuda.cuda.CUDAGraph()
    pipe.scan(x, inclusive=True, out=y, ws=ws)
    cuda.cuda.synchronize()
    with cuda.cuda.graph(g):
        pipe.scan(x, inclusive=True, out=y, ws=ws)
    for _ in range(3):
        y.zero_()
        g.replay()
        assert cuda.equal(y, ref)
    outs = []
    streams = [cuda.cuda.Stream(), cuda.cuda.Stream()]
    cuda.cuda.synchronize()
    for k in range(8):
        with cuda.cuda.stream(streams[k % 2]):
            o, w = cuda.zeros_like(x), pipe.workspace(need)
            pipe.scan(x, inclusive=True, out=o, ws=w)
            outs.append((o, w))
    cuda.cuda.synchronize()
    assert all(cuda.equal(o, ref) for o, _ in outs)
    assert pipe.sync_status() == pipe.EDPP_OK
