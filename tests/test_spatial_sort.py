"""The spatial order of a catalogue by counting (up to 8192 sources) and by radix
passes (tiles of 2048 sources, 256 tiles a step of the scan)."""
import numpy as np
import pytest

from hera_gpu_gb300 import synth, vis_gpu
from oracle import rel_frobenius, vis_oracle

gpu = pytest.mark.gpu


def morton_keys(crd):
    """The sort key in FP32 arithmetic: the octahedral projection of a direction,
    16 bits an axis, interleaved."""
    f = np.float32
    x, y, z = crd
    n = np.abs(x) + np.abs(y) + np.abs(z)
    u, w = x / n, y / n
    south = z < 0
    u, w = (np.where(south, (f(1) - np.abs(w)) * np.where(u < 0, f(-1), f(1)), u),
            np.where(south, (f(1) - np.abs(u)) * np.where(w < 0, f(-1), f(1)), w))
    key = np.zeros(len(x), dtype=np.uint64)
    for axis, v in enumerate((u, w)):
        q = np.clip((v + f(1)) * f(32767.5), f(0), f(65535)).astype(np.uint64)
        for bit in range(16):
            key |= ((q >> np.uint64(bit)) & np.uint64(1)) << np.uint64(2 * bit + axis)
    return key


def catalogue(nant, nsrc, seed):
    """A third of the sources in one direction, another in 50 directions."""
    c = synth.config_array(seed=seed, nant=nant, nsrc=nsrc, ntimes=2, P=15)
    bm = synth.beams_for(c, dtype=np.float32)[0]
    args = [c["antpos"].astype(np.float32), float(c["freqs"][0]), c["eq2tops"].astype(np.float32),
            c["crd_eq"].astype(np.float32), c["I_sky"].astype(np.float32), bm]
    rng = np.random.default_rng(seed)
    shuffled = rng.permutation(nsrc)
    one, some = shuffled[: nsrc // 3], shuffled[nsrc // 3: 2 * nsrc // 3]
    args[3][:, one] = args[3][:, :1]
    args[3][:, some] = args[3][:, rng.integers(0, min(50, nsrc), len(some))]
    return args


# ties in catalogue order on both sides of the switch and of tile edges, in one
# step of the scan and in two; the sum's order is the catalogue's after the sort,
# so one that is in order already gives the same bits
@gpu
@pytest.mark.parametrize("nsrc", [5, 127, 2049, 8189, 8191, 8192, 8193, 10239, 10240, 10241,
                                  600_000])
def test_sources_of_one_key_keep_their_order(nsrc):
    args = catalogue(7, nsrc, seed=nsrc)
    v = vis_gpu(*args, precision=1, method="tc")
    order = np.argsort(morton_keys(args[3]), kind="stable")
    args[3], args[4] = np.ascontiguousarray(args[3][:, order]), args[4][order]
    np.testing.assert_array_equal(vis_gpu(*args, precision=1, method="tc"), v)
    if nsrc <= 20_000:
        ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
        assert rel_frobenius(v, ref).max() <= 1e-4


def test_morton_keys_order_neighbours():
    # (the keys restated here: corners and the fold of the southern half)
    crd = np.array([[0, 0, 1], [0, 0, -1], [1, 0, 0], [-1, 0, 0], [0, 1, 0]], dtype=np.float32).T
    k = morton_keys(crd)
    assert len(set(k.tolist())) == 5 and k.max() < 1 << 32
    assert k[1] == 0xffffffff
