"""Waits of the pipelined scan that run out: the first tile's sum is withheld, so
every block's prefix warps give up after a short limit.  No element is written,
the status says so, and the same arrays scan correctly afterwards.  Lengths with
fewer tiles per block than its ring of 12 buffers (all its copies are issued
before the limit runs out) and with more."""
import pytest

pytestmark = pytest.mark.gpu

TILE = 16384 // 4


@pytest.mark.parametrize("waves", [0.01, 1, 5.5, 12, 13, 40])
def test_withheld_sum(cuda, edpp, waves):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    n = max(1, int(waves * sms * TILE)) + 3
    x = cuda.randint(-9, 9, (n,), dtype=cuda.int32, device="cuda")
    y = cuda.full_like(x, -7)
    ws = edpp.workspace(edpp.scan_workspace_bytes(n, "int32"))
    for _ in range(2):
        edpp.check(edpp.lib().edpp_selftest_scan_pipe_timeout(
            edpp._p(x), edpp._p(y), n, 5_000_000, edpp._p(ws), ws.numel(), edpp._stream()))
        assert edpp.sync_status() == edpp.EDPP_ETIMEOUT
        assert bool((y == -7).all())
    try:
        edpp.tune_set(edpp.TUNE_SCAN_LOOKBACK, 4, n.bit_length() - 1, 3)
        edpp.scan(x, inclusive=True, out=y, ws=ws)
    finally:
        edpp.tune_load(None)
    assert cuda.equal(y, cuda.cumsum(x, 0).to(cuda.int32))
    assert edpp.sync_status() == edpp.EDPP_OK


def test_arguments(cuda, edpp):
    x = cuda.zeros(64, dtype=cuda.int32, device="cuda")
    ws = edpp.workspace(edpp.scan_workspace_bytes(64, "int32"))
    run = lambda i, o, n, t, b: edpp.lib().edpp_selftest_scan_pipe_timeout(  # noqa: E731
        edpp._p(i), edpp._p(o), n, t, edpp._p(ws), b, edpp._stream())
    assert run(x, x, 0, 1, ws.numel()) == edpp.EDPP_EINVAL
    assert run(x, x, 64, 0, ws.numel()) == edpp.EDPP_EINVAL
    assert run(x[1:], x, 8, 1, ws.numel()) == edpp.EDPP_EINVAL
    assert run(x, x[1:], 8, 1, ws.numel()) == edpp.EDPP_EINVAL
    assert run(x, x, 64, 1, 8) == edpp.EDPP_ENOMEM
    assert edpp.sync_status() == edpp.EDPP_OK
