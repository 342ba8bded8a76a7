"""The contexts' workspace under a budget and on a full device, without a GPU
(fake_gpu.py): what a call gets does not depend on the calls before it."""
import ctypes

import numpy as np
import pytest

import fake_gpu
from hera_gpu_gb300 import synth

GB = 1 << 30


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_gpu.build_library(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def gpu(library):
    g = fake_gpu.FakeGpu(library, 280 * GB)
    yield g
    g.close()


# shapes of the calls: precision, method, antennas, sources, times, frequencies
FP32 = (1, "tc", 350, 200_000, 20)
PLAIN = (1, "plain", 350, 100_000, 8)
FP64 = (2, "auto", 350, 100_000, 3)
SIZES = {"tc": FP32, "plain": PLAIN, "fp64": FP64}


# every form after every other one, within a budget that holds each alone: the
# same launches as in a fresh context
@pytest.mark.parametrize("budget", [1 * GB, 2 * GB, 5 * GB])
@pytest.mark.parametrize("first", list(SIZES))
@pytest.mark.parametrize("then", list(SIZES))
def test_a_call_does_not_depend_on_the_one_before(gpu, first, then, budget):
    fresh = gpu.context(budget)
    alone = gpu.call(fresh, *SIZES[then])
    want = fake_gpu.kernels(gpu.log())
    used = gpu.context(budget)
    gpu.call(used, *SIZES[first])
    gpu.log()
    assert gpu.call(used, *SIZES[then]) == alone
    assert fake_gpu.kernels(gpu.log()) == want


# an FP64 call keeps the digit form after a large call in FP32 that fills the budget
def test_fp64_product_after_a_large_fp32_call(gpu):
    ctx = gpu.context(2 * GB)
    assert gpu.call(ctx, *FP32) == 0
    gpu.log()
    assert gpu.call(ctx, 2, "auto", 350, 40_000, 1) == 0
    log = gpu.log()
    assert fake_gpu.launched(log, "mma64_kernel") and not fake_gpu.launched(log, "herk_plain_f64")


# calls that fit as they are allocate, free and wait for nothing
@pytest.mark.parametrize("kind,budget", [("tc", 0), ("tc", 2 * GB), ("plain", 0), ("plain", 1 * GB),
                                         ("plain", 2 * GB), ("fp64", 0), ("fp64", 1 * GB),
                                         ("fp64", 2 * GB), ("fp64", 5 * GB)])
def test_a_repeated_call_keeps_its_workspace(gpu, kind, budget):
    ctx = gpu.context(budget)
    assert gpu.call(ctx, *SIZES[kind]) == 0
    gpu.log()
    gpu.call(ctx, *SIZES[kind])
    assert not [op for op, _, _ in gpu.log() if op in ("malloc", "free", "sync", "hostalloc")]


# nor do they on a device that has room for few slices a launch, or none of the
# digit form
@pytest.mark.parametrize("kind,gb", [("plain", 0.9), ("plain", 1.5), ("plain", 2.2), ("fp64", 0.9),
                                     ("fp64", 1.5), ("fp64", 2.9), ("tc", 2.0)])
def test_a_repeated_call_on_a_small_device(gpu, kind, gb):
    gpu.reset(int(gb * GB))
    ctx = gpu.context()
    assert gpu.call(ctx, *SIZES[kind]) == 0
    gpu.log()
    gpu.call(ctx, *SIZES[kind])
    assert not [op for op, _, _ in gpu.log() if op.split()[0] in ("malloc", "free", "sync")]


# a call whose workspace the one before it has laid out can be captured, also
# where a budget leaves room for few slices a launch, or none of the digit form
@pytest.mark.parametrize("kind", list(SIZES))
@pytest.mark.parametrize("budget", [0] + [(1 << 30) + (k << 26) for k in range(0, 32, 3)])
def test_a_repeated_call_can_be_captured(gpu, kind, budget):
    ctx = gpu.context(budget)
    if gpu.call(ctx, *SIZES[kind], stream=77) != 0:
        return      # a budget below the form's least
    want = fake_gpu.kernels(gpu.log())
    gpu.lib.fake_capture(77)
    assert gpu.call(ctx, *SIZES[kind], stream=77) == 0
    gpu.lib.fake_capture(None)
    log = gpu.log()
    assert fake_gpu.kernels(log) == want
    assert not [op for op, _, _ in log if op.startswith("refused") or op in ("malloc", "free")]


# the FP64 workspace of a captured graph is not given back to a call without room
def test_the_workspace_of_a_captured_call_stays(gpu):
    freed = []
    for captured in (False, True):
        ctx = gpu.context(2 * GB)
        assert gpu.call(ctx, *FP64, stream=77) == 0
        if captured:
            gpu.lib.fake_capture(77)
            assert gpu.call(ctx, *FP64, stream=77) == 0
            gpu.lib.fake_capture(None)
        gpu.log()
        gpu.call(ctx, *FP32)
        freed.append(len([op for op, _, _ in gpu.log() if op == "free"]))
    assert freed[1] <= freed[0] - 4


# small calls fit the budgets that hold one partial sum a 1024 sources and slice
# beside their other workspace (3 % above the least)
@pytest.mark.parametrize("shape,mb", [((1, "tc", 16, 1000, 10), 2.57), ((1, "tc", 64, 3000, 4), 2.96),
                                      ((1, "tc", 350, 3000, 5), 20.8), ((1, "tc", 140, 2000, 8), 10.6),
                                      ((1, "tc", 200, 20_000, 1), 14.8),
                                      ((1, "tc_fp16", 100, 8000, 5), 8.41)])
def test_small_calls_under_a_budget(gpu, shape, mb):
    assert gpu.call(gpu.context(int(mb * 1e6)), *shape, px=31) == 0


# with the room for them they take their shorter chunks, whatever ran before
def test_small_calls_keep_their_chunks(gpu):
    def partial_sums(ctx):      # the largest allocation
        gpu.log()
        assert gpu.call(ctx, 1, "tc", 16, 1000, 10, px=31) == 0
        return max(a for op, a, _ in gpu.log() if op == "malloc")
    fresh = partial_sums(gpu.context())
    assert fresh > 8 * partial_sums(gpu.context(3 << 20))
    used = gpu.context(40 << 20)
    assert gpu.call(used, 1, "plain", 128, 30_000, 1, px=31) == 0
    assert partial_sums(used) >= fresh * 8 // 9


# batches, Omnical, the median filter and device allocations on a device that the
# workspace of an FP64 call has filled
@pytest.mark.parametrize("kind", ["batch", "omnical", "omnical dense", "median", "alloc"])
def test_other_allocations_find_the_workspaces_room(gpu, kind):
    gpu.reset(6 * GB)
    ctx = gpu.context()
    assert gpu.call(ctx, 2, "auto", 350, 60_000, 20) == 0
    left = 6 * GB - gpu.lib.fake_used()
    assert left < 2 * GB        # less than the requests below
    lib = gpu.lib
    if kind == "alloc":
        p = ctypes.c_void_p()
        assert lib.hv_device_alloc(ctx, 3 * GB, ctypes.byref(p)) == 0
    elif kind == "median":
        img = np.zeros((1, 20_000, 16_000), dtype=np.float32)
        assert lib.hv_median_filter(ctx, img.ctypes.data, img.ctypes.data, 1, *img.shape[1:], 3, 3) == 0
    elif kind == "batch":
        assert gpu.batch(ctx, [(350, 60_000, 60, 16)])[0] == 0
    else:
        nants = 100 if kind == "omnical dense" else 20
        ggu, nubls = synth.hex_redundant_layout(nants)
        ggu = np.ascontiguousarray(ggu, dtype=np.uint32)
        n = int(2.2 * GB) // (len(ggu) * 12)
        a = [np.zeros((n, k), dtype=np.complex64) for k in (nants, nubls, len(ggu))]
        w, out = np.zeros((n, len(ggu)), dtype=np.float32), np.zeros((3, n), dtype=np.float32)
        assert lib.hv_omnical(ctx, 1, ggu.ctypes.data, len(ggu), a[0].ctypes.data, nants,
                              a[1].ctypes.data, nubls, a[2].ctypes.data, w.ctypes.data, n, 1e-10, 4,
                              4, 1, 0.3, out[0].ctypes.data, out[1].ctypes.data,
                              out[2].ctypes.data) == 0


# hv_launch_count counts the launches that were made
@pytest.mark.parametrize("shape", [*SIZES.values(), (1, "tc", 350, 3000, 5), (1, "tc", 16, 9000, 2),
                                   (1, "tc_fp16", 200, 5000, 3), (1, "tc", 20, 0, 2),
                                   (2, "auto", 30, 2000, 2), (2, "auto", 2100, 500, 1)])
def test_launches_are_counted(gpu, shape):
    ctx = gpu.context()
    before = gpu.lib.hv_launch_count(ctx)
    assert gpu.call(ctx, *shape) == 0
    assert gpu.lib.hv_launch_count(ctx) - before == len(fake_gpu.kernels(gpu.log()))
