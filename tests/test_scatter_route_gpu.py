"""A scatter takes the direct sweep up to 80% of L2 and the tiled form above;
both sides of the line give the same result as an index assignment."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [-1, 0, 1])
def test_both_sides_of_the_line(cuda, edpp, side):
    lo, hi = 1, 1 << 26
    direct = edpp.lib().edpp_scatter_prefers_direct
    assert direct(lo) and not direct(hi)
    while hi - lo > 1:  # the last length that goes direct
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if direct(mid) else (lo, mid)
    n = lo + side
    g = cuda.Generator(device="cuda")
    g.manual_seed(n)
    loc = cuda.randperm(n, generator=g, device="cuda", dtype=cuda.int32)
    loc[::7] = -1  # skipped: out keeps its value
    inp = cuda.arange(n, dtype=cuda.int32, device="cuda")
    out = cuda.full_like(inp, -5)
    want = out.clone()
    keep = loc >= 0
    want[loc[keep].long()] = inp[keep]
    assert cuda.equal(edpp.scatter(inp, loc, 4, out=out, method="auto"), want)
