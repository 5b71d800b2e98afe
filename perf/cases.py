"""Performance cases: calls that users of the primitives make, over the range of sizes they make them at.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) device inputs, outputs and workspace, as a caller holds them before the call
    run(state)          one call through the public Python entry points
    work(case)          bytes and operations the call cannot do without
    exact(case, seed)   64-bit results of the float cases

Every array is seeded synthetic data made on the GPU.  Outputs and workspaces
are the caller's and kept between calls, which is how the C ABI is used.
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "efficient-dpp_gb300"))

import edpp  # noqa: E402
from edpp import batch as eb  # noqa: E402


def listed():
    return [
        # STREAM triad on float32 at the size the bandwidth figures are quoted on
        dict(name="triad_f32_2p28", kind="stream", op="triad", dtype="float32", n=1 << 28),
        # the smallest scan anyone calls: offsets of a thousand counts, launch latency
        dict(name="scan_i32_1000", kind="scan", dtype="int32", n=1000, inclusive=False,
             algo="lookback"),
        # the plain exclusive prefix sum of 2^24 int32 in [0, 15]
        dict(name="scan_i32_2p24", kind="scan", dtype="int32", n=1 << 24, inclusive=False,
             algo="lookback"),
        # 64-bit offsets, inclusive, reduce-then-scan, a length that ends inside a tile
        dict(name="scan_i64_1e8", kind="scan", dtype="int64", n=100_000_007, inclusive=True,
             algo="rts"),
        # the largest scan: float32 inclusive of 2^30 values in [-1, 1]
        dict(name="scan_f32_2p30", kind="scan", dtype="float32", n=1 << 30, inclusive=True,
             algo="lookback"),
        # gather and scatter of 2^28 int32 through a random permutation, four passes
        dict(name="gather_2p28", kind="gather", n=1 << 28, passes=4),
        dict(name="scatter_2p28", kind="scatter", n=1 << 28, passes=4),
        # a small permutation, as inside a larger pipeline: launch latency
        dict(name="scatter_100003", kind="scatter", n=100_003, passes=4),
        # stable split of 2^28 key/value pairs into 256 buckets, uniform keys
        dict(name="split_soa_256_2p28", kind="split", layout="soa", buckets=256, keys="uniform",
             n=1 << 28, starts=False),
        # a million {key, value} pairs into 16 skewed buckets, with the bucket starts
        dict(name="split_aos_16_1e6", kind="split", layout="aos", buckets=16, keys="zipf",
             n=1_000_003, starts=True),
        # radix sort of key/value pairs over the 31 bits of non-negative keys
        dict(name="radix_kv_2p26", kind="radix", n=1 << 26, values=True),
        # 4096 uneven segments of scan, 64-bucket split and permutation gather in one batch
        dict(name="batch_4096", kind="batch", segments=4096, cap=1 << 30, buckets=64),
    ]


def _log_int(rng, lo, hi):
    """Log-uniform integer in [lo, hi]; every other one is a round power of two."""
    e = rng.uniform(np.log2(lo), np.log2(hi))
    return int(2 ** round(e)) if rng.random() < 0.25 else max(lo, min(hi, int(2.0 ** e)))


def draw(rng):
    kind = rng.choice(["stream", "scan", "scan", "gather", "scatter", "split", "split", "radix",
                       "batch"])
    if kind == "stream":
        return dict(kind=kind, op=rng.choice(["copy", "scale", "add", "triad"]),
                    dtype=rng.choice(["float32", "int32"]), n=_log_int(rng, 1 << 16, 1 << 28))
    if kind == "scan":
        dtype = rng.choice(["int32", "int64", "float32"])
        return dict(kind=kind, dtype=dtype,
                    n=_log_int(rng, 1 << 8, 1 << (28 if dtype == "int64" else 30)),
                    inclusive=rng.random() < 0.5, algo=rng.choice(["lookback", "lookback", "rts"]))
    if kind in ("gather", "scatter"):
        return dict(kind=kind, n=_log_int(rng, 1 << 14, 1 << 28),
                    passes=rng.choice([1, 2, 4, 8, 16]))
    if kind == "split":
        return dict(kind=kind, layout=rng.choice(["ko", "soa", "aos"]),
                    buckets=1 << rng.randint(1, 10), keys=rng.choice(["uniform", "zipf"]),
                    n=_log_int(rng, 1 << 14, 1 << 28), starts=rng.random() < 0.5)
    if kind == "radix":
        return dict(kind=kind, n=_log_int(rng, 1 << 14, 1 << 27), values=rng.random() < 0.5)
    return dict(kind=kind, segments=_log_int(rng, 64, 4096), cap=_log_int(rng, 1 << 24, 1 << 30),
                buckets=1 << rng.randint(2, 8))


# ---- inputs -----------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ints(n, lo, hi, g, dtype=torch.int32):
    """Uniform integers in [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), generator=g, device="cuda", dtype=dtype)


def _floats(n, g):
    """Uniform float32 in [-1, 1)."""
    return torch.rand(n, generator=g, device="cuda").mul_(2).sub_(1)


def _keys(n, kind, buckets, g):
    """Non-negative int32 keys; zipf: bucket b (the low bits) with weight 1 / (b + 1)."""
    k = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64)
    if kind == "zipf":
        w = 1.0 / torch.arange(1, buckets + 1, device="cuda", dtype=torch.float32)
        edges = torch.cumsum(w / w.sum(), 0)[:-1].contiguous()
        u = torch.rand(n, generator=g, device="cuda")
        k = (k & ~(buckets - 1)) | torch.searchsorted(edges, u)
    return k.to(torch.int32)


def _permutation(n, g):
    return torch.randperm(n, generator=g, device="cuda", dtype=torch.int32)


def _scan_input(case, seed):
    g = _gen(seed)
    if case["dtype"] == "float32":
        return _floats(case["n"], g)
    hi = 15 if case["n"] <= 1 << 24 else 100
    return _ints(case["n"], 0, hi, g, getattr(torch, case["dtype"]))


def _stream_input(case, seed):
    g = _gen(seed)
    make = ((lambda: _floats(case["n"], g)) if case["dtype"] == "float32"
            else (lambda: _ints(case["n"], -(1 << 31), (1 << 31) - 1, g)))
    a = make()
    return a, (make() if case["op"] in ("add", "triad") else None)


def _segments(case):
    """The benchmark's 4096-segment size law (log-uniform 2^10..2^24, rescaled to cap)."""
    return eb.config5_segments(num=case["segments"], cap=case["cap"], buckets=case["buckets"])


def _batch_input(segs, seed):
    """in0: values and keys; in1: per-segment permutations of the gathers, values of the splits."""
    g = _gen(seed)
    n = eb.array_length(segs)
    in0 = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    in1 = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    sel = segs[(segs["op"] == eb.OP_GATHER) & (segs["length"] > 0)]
    if len(sel):
        length = torch.from_numpy(sel["length"].astype(np.int64)).cuda()
        offset = torch.from_numpy(sel["offset"].astype(np.int64)).cuda()
        first = torch.cumsum(length, 0) - length
        which = torch.repeat_interleave(torch.arange(len(sel), device="cuda"), length)
        total = which.numel()
        key = (which << 40) | torch.randint(0, 1 << 40, (total,), generator=g, device="cuda",
                                            dtype=torch.int64)
        order = torch.sort(key)[1]  # a random permutation inside each segment
        del key
        pos = torch.arange(total, device="cuda") - first[which] + offset[which]
        in1[pos] = (order - first[which]).to(torch.int32)
    return in0, in1


# ---- one case -----------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "stream":
        s["a"], s["b"] = _stream_input(case, seed)
        s["out"] = torch.empty_like(s["a"])
    elif kind == "scan":
        s["x"] = _scan_input(case, seed)
        s["out"] = torch.empty_like(s["x"])
        s["ws"] = edpp.workspace(edpp.scan_workspace_bytes(case["n"], case["dtype"], case["algo"]))
    elif kind in ("gather", "scatter"):
        g = _gen(seed)
        s["loc"] = _permutation(case["n"], g)
        s["inp"] = _ints(case["n"], -(1 << 31), (1 << 31) - 1, g)
        s["out"] = torch.zeros_like(s["inp"])
        s["ws"] = edpp.workspace(edpp.gs_workspace_bytes(kind, case["n"], case["passes"], "auto"))
    elif kind == "split":
        g = _gen(seed)
        k = _keys(case["n"], case["keys"], case["buckets"], g)
        v = _ints(case["n"], -(1 << 31), (1 << 31) - 1, g) if case["layout"] != "ko" else None
        if case["layout"] == "aos":
            k, v = torch.stack([k, v], dim=1).contiguous(), None
        s["keys"], s["values"] = k, v
        s["keys_out"] = torch.empty_like(k)
        s["values_out"] = torch.empty_like(v) if v is not None else None
        s["ws"] = edpp.workspace(edpp.split_workspace_bytes(case["n"], case["buckets"],
                                                            case["layout"]))
    elif kind == "radix":
        g = _gen(seed)
        s["keys"] = _keys(case["n"], "uniform", 1, g)
        s["values"] = _ints(case["n"], -(1 << 31), (1 << 31) - 1, g) if case["values"] else None
        s["keys_out"] = torch.empty_like(s["keys"])
        s["values_out"] = torch.empty_like(s["keys"]) if case["values"] else None
        s["ws"] = edpp.workspace(edpp.lib().edpp_radix_sort_workspace_size(case["n"],
                                                                           int(case["values"])))
    else:
        segs = _segments(case)
        s["in0"], s["in1"] = _batch_input(segs, seed)
        s["out0"], s["out1"] = torch.zeros_like(s["in0"]), torch.zeros_like(s["in0"])
        s["plan"] = eb.Plan(segs, eb.tuned(segs))
        s["ws"] = s["plan"].workspace()
        s["plan"].upload(s["ws"])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stream":
        return edpp.stream(case["op"], state["a"], state["b"], 3, out=state["out"])
    if kind == "scan":
        return edpp.scan(state["x"], inclusive=case["inclusive"], algo=case["algo"],
                         out=state["out"], ws=state["ws"])
    if kind in ("gather", "scatter"):
        f = edpp.gather if kind == "gather" else edpp.scatter
        return f(state["inp"], state["loc"], case["passes"], out=state["out"], method="auto",
                 ws=state["ws"])
    if kind == "split":
        return edpp.split(state["keys"], case["buckets"], values=state["values"],
                          layout=case["layout"], bucket_start=case["starts"],
                          keys_out=state["keys_out"], values_out=state["values_out"],
                          ws=state["ws"])
    if kind == "radix":
        return edpp.radix_sort(state["keys"], state["values"], 0, 31, keys_out=state["keys_out"],
                               values_out=state["values_out"], ws=state["ws"])
    state["plan"].launch(state["in0"], state["in1"], state["out0"], state["out1"], state["ws"])
    return state["out0"], state["out1"]


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "stream":
        two = case["op"] in ("add", "triad")
        return {"bytes": n * (12 if two else 8), "flops": n * (2 if case["op"] == "triad" else 1)}
    if kind == "scan":
        return {"bytes": n * (16 if case["dtype"] == "int64" else 8), "flops": n}
    if kind in ("gather", "scatter"):
        return {"bytes": n * 12, "flops": 0}
    if kind == "split":
        return {"bytes": n * (8 if case["layout"] == "ko" else 16), "flops": 0}
    if kind == "radix":
        return {"bytes": n * (16 if case["values"] else 8), "flops": 0}
    return {"bytes": eb.algorithmic_bytes(_segments(case)), "flops": 0}


def exact(case, seed):
    if case["kind"] == "scan" and case["dtype"] == "float32":
        x = _scan_input(case, seed).double()
        c = torch.cumsum(x, 0)
        return c if case["inclusive"] else c.sub_(x)
    if case["kind"] == "stream" and case["dtype"] == "float32":
        a, b = _stream_input(case, seed)
        a = a.double()
        return {"copy": lambda: a, "scale": lambda: 3 * a, "add": lambda: a + b.double(),
                "triad": lambda: a + 3 * b.double()}[case["op"]]()
    return None  # whole numbers: equal or wrong
