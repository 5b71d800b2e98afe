"""The one-cluster scan of small inputs at the edges of its tiles (32 and 64 KB)
and cluster sizes (1 to 8 blocks), aligned, off alignment and in place."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("dt", ["int32", "int64", "float32"])
def test_edges(cuda, edpp, dt, algo):
    tdt = getattr(cuda, dt)
    elem = 8 if dt == "int64" else 4
    tile = 32768 // elem
    lengths = [1, 2, 3, 5, 31, 1000]
    for blocks in (1, 2, 3, 7, 8, 10, 16):  # above 8 tiles of 32 KB: 64 KB tiles
        lengths += [blocks * tile - 1, blocks * tile, blocks * tile + 1]
    for n in lengths:
        if dt == "float32":
            # sums of at most 2^18 multiples of 1/8 below 2^3: exact in f32
            x = cuda.randint(-64, 65, (n + 1,), device="cuda").to(tdt) / 8
        else:
            lim = 2**31 if dt == "int32" else 2**62
            x = cuda.randint(-lim, lim - 1, (n + 1,), dtype=tdt, device="cuda")
        for off in (0, 1):  # 1: one element past a 16-byte boundary
            v = x[off:n + off]
            acc = v.double() if dt == "float32" else v.to(cuda.int64)
            ref = cuda.cumsum(acc, 0).to(tdt)  # wraps
            assert cuda.equal(edpp.scan(v, inclusive=True, algo=algo), ref), (n, off)
            assert cuda.equal(edpp.scan(v, algo=algo), ref - v), (n, off)
            w = x.clone()[off:n + off]
            edpp.scan(w, algo=algo, out=w)
            assert cuda.equal(w, ref - v), (n, off)
    assert edpp.sync_status() == edpp.EDPP_OK
