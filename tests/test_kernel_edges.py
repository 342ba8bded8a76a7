"""GPU kernels at the sizes where their launch shapes change: edges of tiles,
remainders, the smallest and largest of a dispatch rule's range, each against
the FP64 oracle on the inputs as the GPU sees them."""
import numpy as np
import pytest

from hera_gpu_gb300 import synth, vis_gpu
from oracle import rel_frobenius, vis_oracle

gpu = pytest.mark.gpu


def sim(nant, nsrc, ntimes=1, P=15, seed=0, dtype=np.float32):
    c = synth.config_array(seed=seed, nant=nant, nsrc=nsrc, ntimes=ntimes, P=P)
    bm = synth.beams_for(c, dtype=dtype)[0]
    return (c["antpos"].astype(dtype), float(c["freqs"][0]), c["eq2tops"].astype(dtype),
            c["crd_eq"].astype(dtype), c["I_sky"].astype(dtype), bm)


def check_hermitian(v):
    np.testing.assert_array_equal(v, np.conj(np.swapaxes(v, -1, -2)))


# split-K reduction: tiles split over four blocks (8 chunks and more: 1024
# sources a chunk in the fused form, 4096 in the plain one) and whole tiles;
# antenna counts at the edges of its 32 x 32 tiles and their 8-column parts
@gpu
@pytest.mark.parametrize("method,tol,nsrc", [("tc", 1e-4, 3000), ("tc", 1e-4, 20000),
                                             ("plain", 1e-5, 5000), ("plain", 1e-5, 33000)])
@pytest.mark.parametrize("nant", [1, 8, 33, 72])
def test_split_k_reduction(nant, nsrc, method, tol):
    args = sim(nant, nsrc, ntimes=2, seed=nant)
    v = vis_gpu(*args, precision=1, method=method)
    check_hermitian(v)
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
    assert rel_frobenius(v, ref).max() <= tol


# spatial sort: one block up to 4096 sources (rows of 512), the radix passes
# beyond (tiles of 2048); any order gives the same sum up to rounding, so a
# lost or doubled source shows as an error far above the tolerance
@gpu
@pytest.mark.parametrize("nsrc", [1, 31, 512, 513, 4095, 4096, 4097, 6144, 6145])
def test_spatial_sort_keeps_every_source(nsrc):
    args = sim(5, nsrc, seed=nsrc)
    args[3][:, : nsrc // 3] = args[3][:, :1]      # ties: many sources in one direction
    v = vis_gpu(*args, precision=1, method="tc")
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
    np.testing.assert_allclose(v, ref, rtol=1e-4, atol=1e-4 * max(1e-30, np.abs(ref).max()))
