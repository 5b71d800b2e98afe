"""A batch launched on a workspace that holds the tables of another plan, whose scan
segments lie off 16-byte alignment: recorded as a plan fault (the pipelined scan
would copy from a misaligned address), nothing written, and the plan's own tables
scan correctly afterwards."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_misaligned_tables(cuda, edpp, shift):
    from edpp import batch
    segs = batch.layout([700 * 4096 - 5] * 7, [batch.OP_SCAN] * 7)
    moved = segs.copy()
    moved["offset"] += shift
    n = batch.array_length(moved)
    x = cuda.randint(-1000, 1000, (n,), dtype=cuda.int32, device="cuda")
    out = cuda.full_like(x, -7)
    plan, other = batch.Plan(segs), batch.Plan(moved)
    ws = plan.workspace("cuda")
    assert other.workspace_bytes == plan.workspace_bytes
    other.upload(ws)
    plan.launch(x, x, out, out, ws)
    assert edpp.sync_status() == edpp.EDPP_EINVAL
    assert bool((out == -7).all())
    plan.upload(ws)
    plan.launch(x, x, out, out, ws)
    assert edpp.sync_status() == edpp.EDPP_OK
    for s in segs:
        o, k = int(s["offset"]), int(s["length"])
        assert cuda.equal(out[o:o + k], (cuda.cumsum(x[o:o + k].long(), 0) - x[o:o + k]).to(cuda.int32))
