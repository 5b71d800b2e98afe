"""Infinities, NaN and sums that overflow in the float scans of every form: one cluster
(each size of 1 to 8 blocks, at the edges of its 32 KB tiles), two launches, the
pipelined scan (below and above one wave of tiles, and one ring of buffers), and the
forms of unaligned arrays.  What lies before a value stays finite, what follows is what
the same sum in 64 bits rounds to; and the error of arrays off 16-byte alignment."""
import pytest

pytestmark = pytest.mark.gpu

TILE = 32768 // 4
INF = float("inf")


@pytest.fixture
def forced(edpp):
    yield lambda prim, variant: (edpp.lib().edpp_tune_clear(), edpp.tune_set(prim, 4, 20, variant))
    edpp.tune_load(None)


def _check(cuda, edpp, n, algo, off):
    for v in (INF, -INF, float("nan"), 3e38):
        for at in sorted({0, 1, n // 3, n // 2 + 1, n - 2} & set(range(n - 1))):
            z = cuda.rand(n + 1, device="cuda")[off:n + off]
            z[at:at + 2] = v
            if v == INF and at + 40 < n:
                z[at + 40] = -INF  # NaN from here on
            ref = cuda.cumsum(z.double(), 0).float()
            out = cuda.empty(n + 1, device="cuda")[off:n + off]
            for inclusive in (True, False):
                y = edpp.scan(z, inclusive=inclusive, algo=algo, out=out)
                r = ref if inclusive else cuda.cat([cuda.zeros(1, device="cuda"), ref[:-1]])
                assert cuda.equal(cuda.isnan(y), cuda.isnan(r)), (n, v, at, inclusive)
                assert cuda.equal(cuda.isposinf(y), cuda.isposinf(r)), (n, v, at, inclusive)
                assert cuda.equal(cuda.isneginf(y), cuda.isneginf(r)), (n, v, at, inclusive)


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("blocks", range(1, 9))
def test_cluster(cuda, edpp, blocks, algo):
    for n in (blocks * TILE - 1, blocks * TILE) + ((blocks * TILE + 1,) if blocks < 8 else ()):
        _check(cuda, edpp, n, algo, 0)
        x = cuda.randint(-2**31, 2**31 - 1, (n + 1,), dtype=cuda.int32, device="cuda")
        for off in (0, 1):
            v = x[off:n + off]
            assert cuda.equal(edpp.scan(v, inclusive=True, algo=algo),
                              cuda.cumsum(v.long(), 0).to(cuda.int32)), (n, off)
    _check(cuda, edpp, blocks * TILE, algo, 1)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("waves", [0.1, 1.5, 13.3])
def test_pipelined(cuda, edpp, forced, waves):
    forced(edpp.TUNE_SCAN_LOOKBACK, 3)
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    _check(cuda, edpp, int(waves * sms * 4096) + 3, "lookback", 0)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("n,off", [(1_000_003, 0), (1_000_003, 1), (13_000_001, 0), (13_000_001, 1)])
def test_two_launches_and_beyond(cuda, edpp, n, off, algo):
    _check(cuda, edpp, n, algo, off)
    assert edpp.sync_status() == edpp.EDPP_OK


@pytest.mark.parametrize("algo", ["lookback", "rts"])
@pytest.mark.parametrize("n", [8 * TILE + 1, 1_000_003, 12_582_912])
def test_error_off_alignment(cuda, edpp, n, algo):
    x = (cuda.rand(n + 1, device="cuda") * 2 - 1)[1:]
    ref = cuda.cumsum(x.double(), 0)
    out = cuda.empty(n + 3, device="cuda")[3:]
    y = edpp.scan(x, inclusive=True, algo=algo, out=out)
    # the two-launch scan's bound, as for aligned arrays: 24 roundings of the sums in a
    # tile and across, two per chunk of four left out of a tile's sum
    lim = 2.0**-24 * (24 * (ref.abs().max().item() + TILE) + 48 * (n / 4)**0.5)
    assert (y.double() - ref).abs().max().item() <= lim
