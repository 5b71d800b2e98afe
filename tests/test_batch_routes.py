"""Which scan kernel a batch takes (host code over a stand-in for the CUDA runtime, no
GPU): the pipelined one for many tiles in long chains, one block per tile for short
segments, whose tiles wait for few others."""
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def fake_lib(edpp, tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


# segments, tiles of each, elements missing from the last: measured us per launch of the
# look-back and of the pipelined kernel
CASES = [
    (65536, 1, 4000, False),  # 204 / 313
    (65536, 1, 0, False),     # 317 / 350
    (8192, 1, 2048, False),   # 33.4 / 50.9
    (4096, 1, 0, False),      # 27.8 / 33.9
    (16384, 4, 0, False),     # 331 / 346
    (2048, 4, 0, False),      # 50.6 / 56.5
    (2048, 16, 0, True),      # 196 / 178
    (256, 16, 0, True),       # 35.8 / 33.2
    (256, 64, 0, True),       # 131 / 98
    (16, 256, 0, True),       # 45.5 / 32.7
    (1, 4095, 0, False),      # too few tiles
]


@pytest.mark.parametrize("segments,tiles,missing,pipe", CASES)
def test_scan_kernel(fake_lib, segments, tiles, missing, pipe):
    got = fake_cuda.run(fake_lib, f"""
import ctypes
import numpy as np
from edpp.batch import SEG_DTYPE
result = []
for shift in (0, 2):
    segs = np.zeros({segments}, SEG_DTYPE)
    segs["length"] = {tiles} * 4096 - {missing}
    segs["offset"] = np.arange({segments}, dtype=np.int64) * ({tiles} * 4096) + shift
    plan = ctypes.c_void_p()
    assert fake.lib.edpp_batch_plan_create(segs.ctypes.data, len(segs), None, ctypes.byref(plan)) == 0
    for off in (0, 4):
        result.append(fake.launches(lambda l: l.edpp_batch_launch(plan, IN + off, IN1, OUT, OUT1, WS, BIG, None)))
    fake.lib.edpp_batch_plan_destroy(plan)
""")
    for k, (status, kernels) in enumerate(got):
        want = "scan_pipe_kernel" if pipe and k == 0 else "kind_scan_kernel"  # aligned, not moved
        assert status == 0 and [x[0] for x in kernels] == [want], k


@pytest.mark.parametrize("ops,asked,blocks", [([0], 0, 4), ([1], 4, 4), ([0, 1, 2], 0, 4), ([2], 0, 3),
                                              ([2, 2], 4, 3), ([1], 3, 3), ([1], 1, 1), ([0, 2], 8, 4)])
def test_queue_blocks_per_sm(fake_lib, ops, asked, blocks):
    """The work-queue kernel: four blocks per SM where asked for, three for gathers alone."""
    status, kernels = fake_cuda.run(fake_lib, f"""
import ctypes
import numpy as np
from edpp.batch import SEG_DTYPE, Tuning
segs = np.zeros(len({ops}), SEG_DTYPE)
segs["length"], segs["op"], segs["buckets"] = 1 << 22, {ops}, 16
segs["offset"] = np.arange(len(segs), dtype=np.int64) << 22
plan, tuning = ctypes.c_void_p(), Tuning({asked}, 1, 1, 1)
assert fake.lib.edpp_batch_plan_create(segs.ctypes.data, len(segs), ctypes.byref(tuning), ctypes.byref(plan)) == 0
result = fake.launches(lambda l: l.edpp_batch_launch(plan, IN, IN1, OUT, OUT1, WS, BIG, None), 0, {max(blocks, 3)})  # what fits of each kernel
""")
    assert status == 0 and len(kernels) == 1
    assert kernels[0][0] == "batch_kernel" and kernels[0][1] == 152 * blocks
    assert f"Li{4 if blocks == 4 else 3}E" in kernels[0][3]
