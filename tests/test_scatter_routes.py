"""The C++ mirror's scatter over a stand-in for the CUDA runtime (no GPU): one direct
sweep while the destination stays in L2, the tiled form beyond and wherever the output
overlaps the input or the indices, which it reads before its first write."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake_lib(edpp, tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


def test_direct_only_without_overlap(fake_lib):
    got = fake_cuda.run(fake_lib, """
import ctypes
f = fake.lib._ZN4edpp10primitives7scatterEPKiPiiS2_iii
f.restype = ctypes.c_double
f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int] * 3
def kernels(src, dst, n, loc):
    return [k[0] for k in fake.launches(lambda l: f(src, dst, n, loc, 0, 0, 4))[1]]
n = 100_003
result = [kernels(IN, OUT, n, LOC), kernels(IN, IN + 4 * n, n, IN + 8 * n), kernels(IN, IN, n, LOC),
          kernels(IN, IN + 4 * n - 4, n, LOC), kernels(IN + 4 * n - 4, IN, n, LOC),
          kernels(IN, LOC, n, LOC), kernels(IN, LOC + 4, n, LOC), kernels(IN, OUT, 1 << 27, LOC)]
""")
    for k in got[:2]:
        assert len(k) == 1 and k[0].startswith("pass_"), k
    for k in got[2:]:
        assert "win_apply_kernel" in k and not any(x.startswith("pass_") for x in k), k
