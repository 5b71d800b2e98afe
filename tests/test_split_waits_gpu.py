"""The wait of the one-launch split that runs out: a block that does not exist is waited
for.  No element is written, the status says so, and the same keys split correctly
afterwards."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,buckets", [(1, 32), (2048, 64), (40_000, 1024), (300_000, 256)])
def test_missing_block(cuda, edpp, n, buckets):
    keys = cuda.randint(0, 2**31 - 1, (n,), dtype=cuda.int32, device="cuda")
    out = cuda.full_like(keys, -7)
    ws = edpp.workspace(edpp.split_workspace_bytes(n, buckets, "ko"))
    for _ in range(2):
        edpp.check(edpp.lib().edpp_selftest_split_timeout(edpp._p(keys), edpp._p(out), n, buckets,
                                                          5_000_000, edpp._p(ws), ws.numel(),
                                                          edpp._stream()))
        assert edpp.sync_status() == edpp.EDPP_ETIMEOUT
        assert bool((out == -7).all())
    edpp.split(keys, buckets, layout="ko", keys_out=out, ws=ws)
    assert cuda.equal(out, keys[cuda.sort(keys & (buckets - 1), stable=True)[1]])
    assert edpp.sync_status() == edpp.EDPP_OK


def test_arguments(cuda, edpp):
    x = cuda.zeros(4096, dtype=cuda.int32, device="cuda")
    y = cuda.zeros_like(x)
    ws = edpp.workspace(edpp.split_workspace_bytes(4096, 256, "ko"))
    run = lambda n, b, t, w: edpp.lib().edpp_selftest_split_timeout(  # noqa: E731
        edpp._p(x), edpp._p(y), n, b, t, edpp._p(ws), w, edpp._stream())
    for n, b, t in ((0, 256, 1), (4096, 16, 1), (4096, 48, 1), (4096, 2048, 1), (4096, 256, 0),
                    (1 << 20, 256, 1)):
        assert run(n, b, t, ws.numel()) == edpp.EDPP_EINVAL
    assert run(4096, 256, 1, 16) == edpp.EDPP_ENOMEM
    assert edpp.sync_status() == edpp.EDPP_OK
