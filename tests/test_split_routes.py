"""Which kernels a split launches (host code over a stand-in for the CUDA runtime, no
GPU): two plain launches while the counts exchanged are few, one cooperative launch
with position staging while they are no more than 2^16, three launches beyond."""
import pytest

import fake_cuda

WORDS, COUNTED = 1 << 16, 1 << 13
FROM = {0: 32, 1: 8, 2: 16}  # position staging: KO, AOS, SOA


@pytest.fixture(scope="module")
def fake_lib(edpp, tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


def _want(n, buckets):
    tiles = lambda t: -(-n // t)
    for t in (2048, 4096, 8192):
        if tiles(t) <= 304 and tiles(t) * buckets <= COUNTED:
            if t == 8192 and tiles(4096) <= 304 and tiles(4096) * buckets <= WORDS:
                break
            return "counted"
    for t, blocks in ((2048, 152), (4096, 152), (8192, 304)):
        if tiles(t) <= blocks and tiles(t) * buckets <= WORDS:
            return "fused"
    return "three"


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_forms(fake_lib, layout):
    cases = [(n, 1 << k) for k in range(11) for n in
             (1, 2048, 2049, 60_000, 152 * 2048, 152 * 2048 + 1, 304 * 2048, 600_001, 152 * 4096,
              304 * 4096 + 1, 2_000_000, 304 * 8192, 304 * 8192 + 1, 5_000_000)]
    got = fake_cuda.run(fake_lib, f"""
result = [[fake.launches(lambda l: l.edpp_split_i32(IN, OUT, LOC, n, b, {layout}, IN1, OUT1, WS, BIG, None), r)[1]
           for r in (0, COOPERATIVE)] for n, b in {cases!r}]
""")
    fused_seen = 0
    for (n, buckets), (plain, refused) in zip(cases, got):
        names = [k[0] for k in plain]
        last = "split_index_kernel" if buckets >= FROM[layout] else "split_scatter_kernel"
        want = _want(n, buckets)
        assert names[-1] == last, (n, buckets)
        if want == "counted":
            assert names == ["split_counts_kernel", last], (n, buckets)
            assert plain[1][2] == fake_cuda.PROGRAMMATIC
        elif want == "fused":
            fused_seen += 1
            assert names == ["split_index_kernel"] and plain[0][2] == fake_cuda.COOPERATIVE
        else:
            assert names[0] == "split_hist_kernel" and len(names) >= 3, (n, buckets)
        if want != "counted":  # refused: three launches
            assert refused[0][0] == "split_hist_kernel" and refused[-1][0] == last, (n, buckets)
    assert fused_seen > 10
