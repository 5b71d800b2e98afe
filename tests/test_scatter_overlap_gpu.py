"""scatter(method="auto") over its own input, over its indices, and over the end of
either: the form chosen reads all of both before it writes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["auto", "tiled"])
@pytest.mark.parametrize("n", [1, 1000, 100_003, (1 << 22) + 1])
def test_overlapping_output(cuda, edpp, n, method):
    g = cuda.Generator(device="cuda")
    g.manual_seed(n)
    loc = cuda.randperm(n, generator=g, device="cuda", dtype=cuda.int32)
    if n > 10:
        loc[n // 3] = -1  # skipped: its element keeps its value
    x = cuda.arange(n, dtype=cuda.int32, device="cuda") * 3 + 1
    ok = loc >= 0

    def want(old):
        w = old.clone()
        w[loc[ok].long()] = x[ok]
        return w

    for _ in range(3):
        y = x.clone()
        edpp.scatter(y, loc, 4, out=y, method=method)
        assert cuda.equal(y, want(x))
        i = loc.clone()
        edpp.scatter(x, i, 4, out=i, method=method)
        assert cuda.equal(i, want(loc))
        for shift in {1, n // 2 + 1, n - 1} - {0, n}:
            for base in (x, loc):  # out starts `shift` elements into it
                both = cuda.cat([base, cuda.full((shift,), -7, dtype=cuda.int32, device="cuda")])
                src, dst = both[:n], both[shift:]
                w = want(dst)
                args = (src, loc) if base is x else (x, src)
                edpp.scatter(*args, 4, out=dst, method=method)
                assert cuda.equal(dst, w), shift
    assert edpp.sync_status() == edpp.EDPP_OK
