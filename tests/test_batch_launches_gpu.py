"""Batches of every subset of the three operations, launched back to back into the
same outputs and workspace and from a CUDA graph: the kernels of one batch start
early beside each other, never beside the batch before."""
import pytest

pytestmark = pytest.mark.gpu

SEGMENTS = 60


@pytest.mark.parametrize("ops", [(0,), (1,), (2,), (0, 1), (0, 2), (1, 2), (0, 1, 2)])
@pytest.mark.parametrize("buckets", [4, 64])
def test_op_subsets_back_to_back(cuda, edpp, ops, buckets):
    import numpy as np

    from edpp import batch as eb

    rng = np.random.default_rng(7)
    segs = np.zeros(SEGMENTS, dtype=eb.SEG_DTYPE)
    segs["length"] = np.where(rng.random(SEGMENTS) < 0.1, 0, 2.0 ** rng.uniform(0, 19, SEGMENTS))
    segs["op"] = [ops[i % len(ops)] for i in range(SEGMENTS)]
    segs["buckets"] = np.where(segs["op"] == eb.OP_SPLIT, buckets, 0)
    n = int(segs["length"].sum()) + 16
    segs["offset"] = np.concatenate([[0], np.cumsum(segs["length"])[:-1]])
    plan = eb.Plan(segs)
    ws = plan.workspace()
    plan.upload(ws)
    sets = []
    for _ in range(3):
        a = cuda.randint(0, 2**30, (n,), dtype=cuda.int32, device="cuda")
        b = cuda.randint(0, 2**30, (n,), dtype=cuda.int32, device="cuda")
        for s in segs[(segs["op"] == eb.OP_GATHER) & (segs["length"] > 0)]:
            o, m = int(s["offset"]), int(s["length"])
            b[o:o + m] = cuda.randperm(m, device="cuda", dtype=cuda.int32)
        want0, want1 = cuda.zeros_like(a), cuda.zeros_like(a)
        for s in segs:
            o, m = int(s["offset"]), int(s["length"])
            x, y = a[o:o + m], b[o:o + m]
            if s["op"] == eb.OP_SCAN:
                want0[o:o + m] = (cuda.cumsum(x.long(), 0) - x).to(cuda.int32)
            elif s["op"] == eb.OP_GATHER:
                want0[o:o + m] = x[y.long()]
            else:
                order = cuda.sort(x & (buckets - 1), stable=True)[1]
                want0[o:o + m], want1[o:o + m] = x[order], y[order]
        sets.append((a, b, want0, want1))
    o0, o1 = cuda.zeros_like(sets[0][0]), cuda.zeros_like(sets[0][0])
    got = []
    for a, b, _, _ in sets:  # no wait between: the copies are on the same stream
        plan.launch(a, b, o0, o1, ws)
        got.append((o0.clone(), o1.clone()))
    for (_, _, w0, w1), (g0, g1) in zip(sets, got):
        assert cuda.equal(g0, w0) and cuda.equal(g1, w1)
    a, b, w0, w1 = sets[0]
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        plan.launch(sets[1][0], sets[1][1], o0, o1, ws)
        plan.launch(a, b, o0, o1, ws)
    for _ in range(3):
        o0.zero_(), o1.zero_()
        graph.replay()
        assert cuda.equal(o0, w0) and cuda.equal(o1, w1)
    assert edpp.sync_status() == edpp.EDPP_OK
