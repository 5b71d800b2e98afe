"""Which kernels a scan launches (host code over a stand-in for the CUDA runtime, no
GPU): the form of every length, whatever the table recorded it, and the forms it
falls back to when a launch is refused."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake_lib(edpp, tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("fn,elem", [("edpp_scan_exclusive_i32", 4), ("edpp_scan_inclusive_i64", 8),
                                     ("edpp_scan_exclusive_f32", 4)])
def test_refused_cluster_launch(fake_lib, fn, elem, algo):
    """A small scan needs no cluster: without one it takes the form of the next sizes,
    and with a workspace off 16 bytes the form of one."""
    got = fake_cuda.run(fake_lib, f"""
result = []
for n in (1, 1000, 65536 // {elem}, (256 << 10) // {elem}):
    for ws in (WS, WS + 8):
        for refuse in (0, CLUSTER):
            result.append(fake.launches(lambda l: l.{fn}(IN, OUT, n, {algo}, ws, BIG, None), refuse))
""")
    for i in range(0, len(got), 4):
        small, refused, small8, refused8 = got[i:i + 4]
        for status, kernels in (small, small8):
            assert status == 0 and [k[0] for k in kernels] == ["scan_small_kernel"]
        assert refused[0] == 0 and [k[0] for k in refused[1]] == ["scan_sums_kernel",
                                                                  "scan_tiles_kernel"]
        assert refused8[0] == 0 and len(refused8[1]) == 1


TABLE = fake_cuda.PKG / "tuning" / "plain_gb300.tsv"
FORMS = {"small": ["scan_small_kernel"], "two": ["scan_sums_kernel", "scan_tiles_kernel"],
         "pipe": ["scan_pipe_kernel"]}


def _form(n, elem):
    if n * elem <= 256 << 10:
        return FORMS["small"]
    return FORMS["two"] if n * elem <= (48 if elem == 4 else 32) << 20 else FORMS["pipe"]


@pytest.mark.parametrize("table", [None, TABLE])
@pytest.mark.parametrize("algo", [0, 1])
def test_form_of_the_length(fake_lib, algo, table):
    """Aligned arrays at the edges of every size class, with the shipped table and
    with none."""
    cases = [(t, n) for t in ("i32", "f32", "i64") for k in range(0, 31)
             for n in ((1 << k) - 1, 1 << k, (1 << k) + 1, 3 << k >> 1) if n]
    for t, elem in (("i32", 4), ("f32", 4), ("i64", 8)):
        top = ((48 if elem == 4 else 32) << 20) // elem
        cases += [(t, n) for n in (top - 1, top, top + 1, (256 << 10) // elem + 1)]
    got = fake_cuda.run(fake_lib, f"""
assert {table is None} or fake.lib.edpp_tune_load({str(table).encode()!r}) == 0
result = [fake.launches(lambda l: getattr(l, "edpp_scan_inclusive_" + t)(IN, OUT, n, {algo}, WS, BIG, None))
          for t, n in {cases!r}]
""")
    for (t, n), (status, kernels) in zip(cases, got):
        assert status == 0 and [k[0] for k in kernels] == _form(n, 8 if t == "i64" else 4), (t, n)


def test_the_table_decides_at_every_length(fake_lib, tmp_path):
    """A recorded variant runs whether it was set, saved and loaded again, or read
    from a caller's file, and edpp_tune_get names it; variant 0 is the form of the
    length."""
    path = str(tmp_path / "t.tsv").encode()
    got = fake_cuda.run(fake_lib, f"""
import ctypes
result = []
def look(n, algo):
    v = ctypes.c_int(-1)
    st = fake.lib.edpp_tune_get(algo, 4, n, ctypes.byref(v))
    return [st, v.value, [k[0] for k in fake.launches(
        lambda l: l.edpp_scan_exclusive_i32(IN, OUT, n, algo, WS, BIG, None))[1]]]
for n in (1000, 100_000, 5_000_000, 25_000_000):
    for algo in (0, 1):
        for variant in (0, 1):
            fake.lib.edpp_tune_clear()
            cls = n.bit_length() - 1
            assert fake.lib.edpp_tune_set(algo, 4, cls, variant, 0.0) == 0
            seen = [look(n, algo)]
            assert fake.lib.edpp_tune_save({path!r}) == 0
            fake.lib.edpp_tune_clear()
            seen.append(look(n, algo))
            assert fake.lib.edpp_tune_load({path!r}) == 0
            seen.append(look(n, algo))
            result.append([n, algo, variant, seen])
""")
    for n, algo, variant, (was_set, cleared, loaded) in got:
        assert was_set == loaded and was_set[:2] == [0, variant]
        assert cleared == [1, 0, _form(n, 4)]
        if variant == 0:
            assert was_set[2] == _form(n, 4)
        elif algo == 0:
            assert was_set[2] == ["scan_lookback_kernel"]
        else:
            assert was_set[2] == ["rts_fused_kernel" if n < 15_000_000 else "rts_chunked_kernel"]


def test_workspace_off_16_bytes(fake_lib):
    got = fake_cuda.run(fake_lib, """
result = [[n, algo] + fake.launches(lambda l: l.edpp_scan_exclusive_i32(IN, OUT, n, algo, WS + 8, BIG, None))[1][-1:]
          for n in (100_000, 1 << 19, (1 << 19) + 1, 1 << 23, 1 << 25) for algo in (0, 1)]
""")
    for n, algo, (kernel, *_) in got:
        small = "scan_lookback_kernel" if algo == 0 else "rts_fused_kernel"
        assert kernel == (small if n <= 1 << 19 else "scan_pipe_kernel"), (n, algo)


@pytest.mark.parametrize("t,elem", [("i32", 4), ("f32", 4), ("i64", 8)])
def test_slices_of_unaligned_reduce_then_scan(fake_lib, t, elem):
    """Slices of four tiles from 256 MB on where only the output is off 16 bytes."""
    line = (256 << 20) // elem
    got = fake_cuda.run(fake_lib, f"""
result = [fake.launches(lambda l: l.edpp_scan_exclusive_{t}(IN + i * {elem}, OUT + o * {elem}, n, 1, WS, BIG, None))
          for n in ({line} - 1, {line}, 4 * {line} + 3) for i, o in ((1, 0), (0, 1), (1, 1))]
""")
    for k, (status, kernels) in enumerate(got):
        assert status == 0 and [x[0] for x in kernels] == ["rts_chunked_kernel"]
        four = k % 3 == 1 and k > 3
        assert ("ELi4E" if four else "ELi2E") in kernels[0][3], (k, kernels)
