"""A scan variant recorded by edpp_tune_set is what runs, also at the sizes that
otherwise do not ask the table."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 100_003])
@pytest.mark.parametrize("algo", ["lookback", "rts"])
def test_set_variant_runs_at_any_size(cuda, edpp, algo, n):
    prim = edpp.TUNE_SCAN_LOOKBACK if algo == "lookback" else edpp.TUNE_SCAN_RTS
    x = cuda.randint(-9, 9, (n,), dtype=cuda.int32, device="cuda")
    ref = cuda.cumsum(x, 0).to(cuda.int32)

    # the table's variants zero all of it; the one-cluster form leaves it alone and
    # the two-launch form writes a sum per 32 KB tile (13 words at 100003)
    def header():
        ws = edpp.workspace(edpp.scan_workspace_bytes(n, "int32", algo))
        ws.view(cuda.uint8).fill_(0xAB)
        assert cuda.equal(edpp.scan(x, inclusive=True, algo=algo, ws=ws), ref)
        return ws.view(cuda.uint8)[:256].clone()

    try:
        assert edpp.tune_load(None) == edpp.EDPP_OK
        assert (header()[128:] == 0xAB).all()
        edpp.tune_set(prim, 4, max(n.bit_length() - 1, 0), 1)
        assert (header() != 0xAB).all()
    finally:
        edpp.tune_load(None)
    assert edpp.sync_status() == edpp.EDPP_OK
