"""The streams of a batch's size classes, without a GPU (fake_gpu.py)."""
import ctypes

import pytest

import fake_gpu

SIMS = [(16, 1000, 2, 1), (150, 2000, 2, 1), (300, 3000, 2, 1), (90, 500, 1, 1), (60, 500, 1, 1)]


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_gpu.build_library(tmp_path_factory.mktemp("fake"))


@pytest.fixture
def gpu(library):
    g = fake_gpu.FakeGpu(library, 64 << 30)
    yield g
    g.close()


def fused(log):
    """(position, stream) of the fused kernel's launches."""
    return [(i, a) for i, (op, a, _) in enumerate(log) if op.startswith("launch ")
            and "tc_vis_kernel" in op]


# with profiling on, the sum of the classes' times is time on one stream: none
# begins before the one before it has ended
def test_profiled_classes_do_not_overlap(gpu):
    ctx = gpu.context()
    rc, batch = gpu.batch(ctx, SIMS)
    assert rc == 0
    assert len({s for _, s in fused_launch(gpu, batch)}) > 1
    gpu.lib.hv_set_profiling(ctx, 1)
    gpu.log()
    assert gpu.lib.hv_batch_launch(batch, None) == 0
    log = gpu.log()
    timed = [(i, a) for i, (op, a, _) in enumerate(log) if op == "eventcreate"]
    assert len(timed) == 2 * len(SIMS)
    events = {a for _, a in timed}
    assert len({s for op, e, s in log if op == "record" and e in events}) == 1
    ms, n = ctypes.c_double(), ctypes.c_uint64()
    assert gpu.lib.hv_profile_read(ctx, ctypes.byref(ms), ctypes.byref(n)) == 0
    assert n.value == len(SIMS)
    gpu.lib.hv_batch_destroy(batch)


def fused_launch(gpu, batch):
    gpu.log()
    assert gpu.lib.hv_batch_launch(batch, None) == 0
    return fused(gpu.log())


# a launch that fails between the fork and the join: what the other streams were
# given is waited for before the arena is given back on the batch's stream
@pytest.mark.parametrize("after", [1, 2, 3, 4])
def test_a_failed_class_joins_its_streams(gpu, after):
    ctx = gpu.context()
    rc, batch = gpu.batch(ctx, SIMS)
    assert rc == 0
    gpu.log()
    gpu.lib.fake_fail(b"tc_vis_kernel", after)
    assert gpu.lib.hv_batch_launch(batch, None) != 0
    gpu.lib.hv_batch_destroy(batch)
    log = gpu.log()
    freed = next(i for i, (op, _, _) in enumerate(log) if op == "freeasync")
    own = log[freed][1]
    last = {s: i for i, s in fused(log[:freed]) if s != own}
    assert last
    for stream, i in last.items():
        joined = [e for j, (op, e, s) in enumerate(log[:freed]) if j > i and op == "record" and s == stream]
        assert any(op == "wait" and s == own and e in joined for op, s, e in log[i:freed])
