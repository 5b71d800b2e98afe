"""Which kernels a scan launches (host code over a stand-in for the CUDA runtime, no
GPU): the forms it falls back to when a launch is refused."""
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
