"""The tiled gather of requests that lie close together, which the group kernel reads
directly: by their span, by their vectors, or by the window that all tiles around read;
next to grouped tiles, with invalid indices, off 16-byte alignment, and with arrays
that overlap, where no tile may be read directly."""
import pytest

pytestmark = pytest.mark.gpu

TILE, NEAR, NEAR_ALL = 8192, 65536, 1 << 23


def _loc(cuda, kind, n):
    g = cuda.Generator(device="cuda")
    g.manual_seed(n)
    i = cuda.arange(n, device="cuda")
    rand = cuda.randint(0, n, (n,), generator=g, device="cuda")
    if kind == "identity":
        return i
    if kind == "one":
        return cuda.full_like(i, n - 1)
    if kind == "rows":  # of 64 elements, in random order
        m = n // 64
        return cuda.cat([(cuda.randperm(m, generator=g, device="cuda")[:, None] * 64
                          + cuda.arange(64, device="cuda")).flatten(), i[m * 64:]])
    if kind == "window":
        return rand % min(n, NEAR_ALL)
    if kind == "wide_window":
        return rand % min(n, 2 * NEAR_ALL)
    if kind == "none_valid":
        return cuda.where(i % 2 == 0, i - n, i + n)
    near = (i // TILE * TILE + rand % (NEAR - TILE)).clamp(max=n - 1)
    if kind == "near":
        return near
    if kind == "edge":  # spans of exactly NEAR - 1, NEAR and NEAR + 1 in turn
        return cuda.where(i % TILE == 4097, i // TILE * TILE + NEAR - 1 + i // TILE % 3,
                          i // TILE * TILE).clamp(max=n - 1)
    assert kind == "mixed"  # tiles near, grouped, invalid and half in rows, in turn
    t = i // TILE % 4
    out = cuda.where(t == 0, near, rand)
    out = cuda.where(t == 2, -1, out)
    return cuda.where((t == 3) & (i % TILE < 5000), i, out)


KINDS = ["identity", "one", "rows", "window", "wide_window", "none_valid", "near", "edge", "mixed"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [1, 5, TILE, 20 * TILE + 3, (1 << 24) + 1, (1 << 25) + 4097])
def test_near_requests(cuda, edpp, n, kind):
    loc = _loc(cuda, kind, n)
    loc[n // 2] = -2**31  # skipped
    x = cuda.arange(n, dtype=cuda.int32, device="cuda") * 3 + 1
    old = cuda.full_like(x, -7)
    ok = (loc >= 0) & (loc < n)
    want = cuda.where(ok, x[loc.clamp(0, n - 1)], old)
    loc = loc.to(cuda.int32)
    assert cuda.equal(edpp.gather(x, loc, 4, out=old.clone(), method="tiled"), want)
    for a in (0, 1):  # out and loc off 16-byte alignment, in turn
        o, l = cuda.full((n + 1,), -7, dtype=cuda.int32, device="cuda"), cuda.empty(n + 1, dtype=cuda.int32, device="cuda")
        l[1 - a:n + 1 - a] = loc
        got = edpp.gather(x, l[1 - a:n + 1 - a], 4, out=o[a:n + a], method="tiled")
        assert cuda.equal(got, want)
    # in place, over loc, and over the middle of both
    y = x.clone()
    edpp.gather(y, loc, 4, out=y, method="tiled")
    assert cuda.equal(y, cuda.where(ok, want, x))
    l = loc.clone()
    edpp.gather(x, l, 4, out=l, method="tiled")
    assert cuda.equal(l, cuda.where(ok, want, loc))
    h = n // 2
    both = cuda.cat([x, cuda.full((h,), -7, dtype=cuda.int32, device="cuda")])
    src, dst = both[:n], both[h:h + n]
    keep = dst.clone()
    edpp.gather(src, loc, 4, out=dst, method="tiled")
    assert cuda.equal(dst, cuda.where(ok, want, keep))
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("kind,direct", [("identity", True), ("rows", True), ("near", True),
                                         ("window", True), ("wide_window", False)])
def test_near_tiles_are_not_grouped(cuda, edpp, kind, direct):
    """A tile read directly leaves its stretch of the workspace (the requests, 4 bytes
    each) alone; a grouped one fills it."""
    n = (1 << 25) + TILE
    loc = _loc(cuda, kind, n).to(cuda.int32)
    x = cuda.arange(n, dtype=cuda.int32, device="cuda")
    ws = edpp.workspace(edpp.gs_workspace_bytes("gather", n, 4, "tiled")).view(cuda.uint8)
    ws.fill_(0xAB)
    assert cuda.equal(edpp.gather(x, loc, 4, method="tiled", ws=ws), loc)
    left = (ws[:4 * n].view(cuda.int32).view(-1, TILE) == 0xABABABAB - (1 << 32)).all(1)
    assert left.float().mean() > 0.99 if direct else not left.any()
