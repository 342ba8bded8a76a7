"""The antenna-matrix kernel of float32 Omnical against the general kernel, which
solves the same problem when a pair is listed once more with weight zero."""
import numpy as np
import pytest

import fake_gpu
from hera_gpu_gb300 import omnical, synth
from oracle import omnical_oracle

gpu = pytest.mark.gpu


def problem(nants, ndata, seed):
    ggu, nubls = synth.hex_redundant_layout(nants)
    g0, u0, d, w = synth.redundant_data(ggu, nubls, ndata, seed=seed, noise=0.02)
    return ggu, [x.astype(t) for x, t in ((g0, np.complex64), (u0, np.complex64),
                                          (d, np.complex64), (w, np.float32))]


# both round about as often, so their distances from the 64-bit iteration agree
# within a few percent over 100 problems; sums of many terms added one after
# the other would put the antenna-matrix kernel's a quarter above
@gpu
@pytest.mark.parametrize("nants", [33, 53, 92, 128, 150])
def test_errors_are_no_larger_than_the_general_kernels(nants):
    ggu, a = problem(nants, 100, seed=nants)
    dense = omnical(ggu, *a, 1e-10, 12, precision=1)
    again = np.concatenate([ggu, ggu[:1]])
    b = a[:2] + [np.concatenate([a[2], a[2][:, :1]], 1),
                 np.concatenate([a[3], np.zeros_like(a[3][:, :1])], 1)]
    general = omnical(again, *b, 1e-10, 12, precision=1)
    ref = omnical_oracle(ggu, *[x.astype(np.complex128 if np.iscomplexobj(x) else np.float64)
                                for x in a], 1e-10, 12, precision=2)
    for x in ("gains", "ubls"):
        far = [np.linalg.norm(v[x] - ref[x]) for v in (dense, general)]
        assert far[0] <= 1.1 * far[1], (x, far)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    g = fake_gpu.FakeGpu(fake_gpu.build_library(tmp_path_factory.mktemp("fake")), 64 << 30)
    yield g
    g.close()


# the antenna-matrix kernel is taken only where it was measured to be no slower,
# whatever the number of problems: full hexagons (no count of unique baselines),
# and layouts with more unique baselines
@pytest.mark.parametrize("nants,nubls,dense", [
    (30, None, 0), (31, None, 1), (54, None, 1), (64, None, 1), (65, None, 0), (80, None, 0),
    (84, None, 0), (87, None, 0), (88, None, 1), (128, None, 1), (180, None, 1), (256, None, 1),
    (257, None, 0), (31, 160, 0), (48, 264, 0), (54, 147, 1), (54, 196, 0), (64, 178, 1),
    (64, 357, 0), (96, 277, 1), (96, 370, 0), (112, 632, 1), (128, 723, 1), (128, 800, 0),
    (150, 568, 1), (150, 852, 0), (180, 522, 1), (180, 800, 0), (225, 872, 1), (256, 980, 1)])
def test_which_kernel_a_layout_takes(fake, nants, nubls, dense):
    ggu, full = synth.hex_redundant_layout(nants)
    ggu = ggu.astype(np.uint32)
    if nubls:
        own = np.random.default_rng(1).permutation(len(ggu))[: nubls - full]
        ggu[own, 2] = full + np.arange(len(own))
    n_u = int(ggu[:, 2].max()) + 1
    ggu = np.ascontiguousarray(ggu)
    ctx = fake.context()
    for ndata in (1, 3000):
        dev = 1 << 20
        assert fake.lib.hv_omnical_device(ctx, 1, ggu.ctypes.data, len(ggu), dev, nants, dev, n_u, dev,
                                          dev, ndata, 1e-10, 12, 4, 1, 0.3, dev, dev, dev, None) == 0
        log = fake.log()
        assert fake_gpu.launched(log, "omnical_dense_kernel") == dense
        assert fake_gpu.launched(log, "omnical_kernel") == 1 - dense
