"""The tile-local gather at the edges of its tiles (8192), of its rows of
tiles (32) and of its window sizes, with repeated, skewed and invalid indices,
unaligned arrays and in place."""
import numpy as np
import pytest

from conftest import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["uniform", "one_window", "sorted"])
@pytest.mark.parametrize("n", [1, 3, 1024, 8191, 8192, 8193, 65 * 1024, 32 * 8192 - 1, 32 * 8192,
                               33 * 8192 + 5, (1 << 22) + 1])
def test_edges(cuda, edpp, orc, n, kind):
    rng = np.random.default_rng(n)
    if kind == "uniform":
        loc = rng.integers(-3, n + 3, n)
    elif kind == "one_window":
        loc = rng.integers(0, min(n, 700), n)
    else:
        loc = np.sort(rng.integers(0, n, n))
    loc = loc.astype(np.int32)
    if n > 3:
        loc[1], loc[2] = -2**31, 2**31 - 1
    inp = rng.integers(-2**31, 2**31, n).astype(np.int32)
    out0 = np.full(n, 99, np.int32)
    want = orc.gather(inp, loc, 1, out=out0)
    got = edpp.gather(to_dev(inp), to_dev(loc), 4, out=to_dev(out0), method="tiled")
    np.testing.assert_array_equal(to_host(got), want)
    # arrays one element past a 16-byte boundary
    pad = lambda a: to_dev(np.concatenate([np.zeros(1, np.int32), a]))[1:]
    got = edpp.gather(pad(inp), pad(loc), 4, out=pad(out0), method="tiled")
    np.testing.assert_array_equal(to_host(got), want)
    # in place: every read of the source precedes the first write
    x = to_dev(inp)
    edpp.gather(x, to_dev(loc), 4, out=x, method="tiled")
    np.testing.assert_array_equal(to_host(x), orc.gather(inp, loc, 1, out=inp.copy()))
    assert edpp.sync_status() == edpp.EDPP_OK
