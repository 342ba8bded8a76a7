"""The antenna-matrix kernel of float32 Omnical against the general kernel, which
solves the same problem when a pair is listed once more with weight zero."""
import numpy as np
import pytest

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
@pytest.mark.parametrize("nants", [33, 53, 84, 128, 150])
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
