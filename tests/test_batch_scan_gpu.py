"""Batched scans above and below the tile count that takes the pipelined scan
(4096 tiles of 4096 elements): segments of one element, of one tile, ragged and long
ones, so that heads fall everywhere in a wave; unaligned offsets keep the
tile-per-block kernel; graph replay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PIPE_TILES = 4096


def _lengths(kind, tiles):
    if kind == "short":  # a head in every word of a wave
        return [1 + (i * 7) % 4096 for i in range(tiles)]
    if kind == "long":
        return [tiles * 4096 - 5]
    rng = np.random.default_rng(tiles)
    out, left = [], tiles
    while left > 0:
        t = int(min(left, rng.choice([1, 1, 2, 3, 151, 152, 153, 304, 700])))
        out.append(t * 4096 - int(rng.choice([0, 1, 2, 3, 4095])))
        left -= t
    return out


def _want(cuda, segs, x):
    c = cuda.cumsum(x.to(cuda.int64), 0)
    out = cuda.zeros_like(x)
    for s in segs:
        o, n = int(s["offset"]), int(s["length"])
        before = c[o - 1] if o else 0
        out[o:o + n] = (c[o:o + n] - x[o:o + n] - before).to(cuda.int32)
    return out


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("tiles", [PIPE_TILES - 1, PIPE_TILES, 9001])
@pytest.mark.parametrize("kind", ["short", "mixed", "long"])
def test_scan_segments(cuda, edpp, kind, tiles, shift):
    from edpp import batch
    segs = batch.layout(_lengths(kind, tiles), [batch.OP_SCAN] * len(_lengths(kind, tiles)))
    segs["offset"] += shift  # 1: off the 16-byte boundary
    n = batch.array_length(segs)
    x = cuda.randint(-1000, 1000, (n + 8,), dtype=cuda.int32, device="cuda")
    out = cuda.zeros_like(x)
    plan = batch.Plan(segs)
    ws = plan.workspace("cuda")
    plan.upload(ws)
    want = _want(cuda, segs, x)
    plan.launch(x, x, out, out, ws)
    assert cuda.equal(out, want)
    g = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g):
        plan.launch(x, x, out, out, ws)
    out.zero_()
    g.replay()
    assert cuda.equal(out, want)
    assert edpp.sync_status() == edpp.EDPP_OK
