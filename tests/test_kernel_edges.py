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


# FP64 product on the tensor cores.  Each entry is compared relative to
# sqrt(V_aa V_bb), the scale FP64 rounding acts on, so that an antenna with a
# faint beam is held to the same relative error.  1e-11 is the FP64 path's
# bound (phases of up to ~1e3 cycles rounded in FP64: 1e3 * 2^-53 * 2 pi).
F64_TOL = 1e-11


def oracle64(args):
    return vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])


def check64(v, ref):
    p = np.sqrt(np.abs(np.einsum("taa->ta", ref)))
    scale = p[:, :, None] * p[:, None, :]
    assert np.all(np.abs(v - ref) <= F64_TOL * scale + 1e-300)


# one to three antenna blocks; sources around the 32-source steps
@gpu
@pytest.mark.parametrize("nant,nsrc", [(1, 1), (2, 63), (32, 65), (33, 500), (127, 4200),
                                       (128, 130), (129, 1000), (300, 700), (7, 0)])
def test_fp64_product(nant, nsrc):
    args = sim(nant, nsrc, ntimes=2, seed=nant + nsrc, dtype=np.float64)
    v = vis_gpu(*args, precision=2)
    check_hermitian(v)
    check64(v, oracle64(args))


# more than one window of 65536 sources above the horizon
@gpu
def test_fp64_product_source_windows():
    args = sim(5, 150_000, ntimes=1, seed=3, dtype=np.float64)
    v = vis_gpu(*args, precision=2)
    check_hermitian(v)
    check64(v, oracle64(args))


# several launches of whole times, and of some frequencies of one time, must
# give the bits of one launch: a budget leaves room for fewer slices, or for
# none (the SIMT product: other rounding)
@gpu
def test_fp64_product_under_a_budget():
    from hera_gpu_gb300 import vis_gpu_multifreq
    from hera_gpu_gb300._native import Context
    c = synth.config_array(seed=4, nant=130, nsrc=3000, ntimes=3, nfreq=3, fmin=1e8, fmax=2e8, P=9)
    bm = synth.beams_for(c, dtype=np.float64)
    args = (c["antpos"], c["freqs"], c["eq2tops"], c["crd_eq"], c["I_sky"], bm)
    full = vis_gpu_multifreq(*args, precision=2)
    for mb, same in ((120, True), (60, True), (33, False)):
        v = vis_gpu_multifreq(*args, precision=2, context=Context(0, hbm_budget_bytes=mb << 20))
        if same:
            np.testing.assert_array_equal(v, full)
        else:
            assert np.abs(v - full).max() <= F64_TOL * np.abs(full).max()


# phases in fixed point: arrays from a micrometre to a light second.  Both
# sides round U and the oracle its phase sums in FP64: 8 roundings of the
# largest |U| in cycles, and 1e-14 for the amplitudes
@gpu
@pytest.mark.parametrize("scale", [1e-8, 1e-3, 1.0, 1e3, 1e6])
def test_fp64_phases(scale):
    args = list(sim(24, 700, ntimes=2, seed=7, dtype=np.float64))
    args[0] = args[0] * scale
    v = vis_gpu(*args, precision=2)
    check_hermitian(v)
    cycles = np.sqrt((args[0] ** 2).sum(axis=1)).max() * args[1] / 299792458.0
    tol = 1e-14 + 2 * np.pi * 8 * 2.0 ** -53 * cycles
    assert rel_frobenius(v, vis_oracle(*args)).max() <= tol


# phases of 2^56 cycles and more carry no information, but stay phases: the
# autocorrelations do not know them
@gpu
def test_fp64_phases_beyond_fixed_point():
    args = list(sim(24, 700, ntimes=2, seed=7, dtype=np.float64))
    near = vis_gpu(*args, precision=2)
    args[0] = args[0] * 2.0 ** 60
    v = vis_gpu(*args, precision=2)
    check_hermitian(v)
    np.testing.assert_allclose(np.einsum("taa->ta", v), np.einsum("taa->ta", near), rtol=1e-13)


# antennas of very different scale, a dark antenna, and scales outside the
# digit form's range (2^-400): the slice takes the SIMT product
@gpu
@pytest.mark.parametrize("small", [1e-30, 1e-100, 1e-140])
def test_fp64_product_antenna_scales(small):
    args = list(sim(40, 900, ntimes=1, seed=5, dtype=np.float64))
    bm = args[5].copy()
    bm[3] *= small
    bm[17] = 0.0
    bm[21] *= -1.0
    args[5] = bm
    v = vis_gpu(*args, precision=2)
    check64(v, oracle64(args))
    np.testing.assert_array_equal(v[0, 17], 0)


# infinities and NaN reach the entries they reach in the SIMT product
@gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_fp64_product_not_finite(bad):
    args = list(sim(35, 400, ntimes=2, seed=6, dtype=np.float64))
    clean = vis_gpu(*args, precision=2)
    bm = args[5].copy()
    bm[4] = bad
    args[5] = bm
    v = vis_gpu(*args, precision=2)
    others = [a for a in range(35) if a != 4]
    assert not np.isfinite(v[:, 4]).any() and not np.isfinite(v[:, :, 4]).any()
    np.testing.assert_allclose(v[:, others][:, :, others], clean[:, others][:, :, others],
                               rtol=0, atol=F64_TOL * np.abs(clean).max())


# median strip kernels: every window shape they take (and the nearest they do
# not), images narrower than a window, at the edges of the strips (128 columns
# for 3 x 3, 52 to 62 otherwise) and of their 16 rows, with signed zeros,
# infinities, NaN and ties
@gpu
@pytest.mark.parametrize("ks", [(h, w) for h in (1, 3, 5, 7, 9) for w in (1, 3, 5, 7, 9)]
                         + [(1, 11), (11, 1), (11, 3), (2, 3)])
def test_median_strips(ks):
    from hera_gpu_gb300 import MedianFilter
    from oracle import median_filter_oracle
    rng = np.random.default_rng(ks[0] * 16 + ks[1])
    for shape in ((1, 1), (2, 3), (15, 52), (16, 54), (17, 63), (33, 129), (40, 260)):
        img = rng.normal(size=shape).astype(np.float32)
        img[rng.random(shape) < 0.2] = 0.0
        img[rng.random(shape) < 0.1] = -0.0
        img[rng.random(shape) < 0.1] = 1.0
        img[rng.random(shape) < 0.03] = np.inf
        img[rng.random(shape) < 0.03] = -np.inf
        out = MedianFilter(input=img, kernel_size=ks)[0]
        ref = median_filter_oracle(img, *ks)
        np.testing.assert_array_equal(out, ref)          # zeros compare equal whatever their sign
    # keys order -0.0 below 0.0 and NaN by its bits: a window of NaN is NaN
    img[:] = np.nan
    inner = MedianFilter(input=img, kernel_size=ks)[0][8:-8, 8:-8]
    assert np.isnan(inner).all()


# omnical in float32: the antenna-matrix kernel (31 to 64 and 80 to 256 antennas,
# distinct pairs) at the edges of its rows and column chunks, with pairs in both orders,
# baselines in any order and some missing; and layouts it must leave to the
# general kernel (fewer, 65 to 79 and 257 antennas, a pair twice, one unique
# baseline for all).  A dozen iterations: float32 rounding (6e-8 a step and term) stays far
# below 1e-5 of the largest gain, and no problem is near a stop.
@gpu
@pytest.mark.parametrize("nants", [16, 17, 30, 31, 32, 33, 64, 65, 79, 80, 96, 97, 128, 129, 192,
                                   193, 256, 257])
@pytest.mark.parametrize("kind", ["plain", "shuffled", "twice", "one"])
def test_omnical_layouts(nants, kind):
    from hera_gpu_gb300 import omnical
    from oracle import omnical_oracle
    if kind != "plain" and nants not in (17, 64, 129, 193):
        pytest.skip("the other layouts at one size of each launch shape")
    ggu, nubls = synth.hex_redundant_layout(nants)
    rng = np.random.default_rng(nants)
    if kind == "one":       # the same unique baseline many times in a row
        ggu = ggu.copy()
        ggu[:, 2] = 0
        nubls = 1
    g0, u0, d, w = synth.redundant_data(ggu, nubls, 3, seed=nants, noise=0.05)
    if kind == "shuffled":
        keep = rng.permutation(len(ggu))[: len(ggu) * 9 // 10]
        keep = np.unique(np.concatenate([keep, [np.flatnonzero(ggu[:, 2] == k)[0] for k in range(nubls)]]))
        keep = rng.permutation(keep)
        ggu, d, w = ggu[keep], d[:, keep], w[:, keep]
        swap = rng.random(len(ggu)) < 0.5
        ggu = ggu.copy()
        ggu[swap] = ggu[swap][:, [1, 0, 2]]
        d[:, swap] = np.conj(d[:, swap])     # the model of (j, i) with the same unique baseline:
        # conj(g_i) g_j u differs from conj(g_i conj(g_j) u) by u's phase, so give the pair its own
        # consistent data
        d[:, swap] = d[:, swap] * np.exp(2j * np.angle(u0[:, ggu[swap, 2]]))
    if kind == "twice":
        ggu = np.concatenate([ggu, ggu[:1]])
        d, w = np.concatenate([d, d[:, :1]], 1), np.concatenate([w, w[:, :1]], 1)
    a = [x.astype(t) for x, t in ((g0, np.complex64), (u0, np.complex64), (d, np.complex64),
                                  (w, np.float32))]
    got = omnical(ggu, *a, 1e-10, 12, precision=1)
    ref = omnical_oracle(ggu, *a, 1e-10, 12, precision=1)
    assert np.abs(got["gains"] - ref["gains"]).max() <= 1e-5 * np.abs(ref["gains"]).max()
    assert np.abs(got["ubls"] - ref["ubls"]).max() <= 1e-5 * np.abs(ref["ubls"]).max()
    np.testing.assert_allclose(got["chisq"], ref["chisq"], rtol=1e-3)
    np.testing.assert_array_equal(got["iters"], ref["iters"])
    again = omnical(ggu, *[x[1:] for x in a], 1e-10, 12, precision=1)
    np.testing.assert_array_equal(again["gains"], got["gains"][1:])


# omnical in float64: everything in shared memory (data times weights kept), and
# panels of baselines, with flagged samples.  A dozen iterations of 1e-16 a step
# and term stay far below 1e-11 of the largest gain
@gpu
@pytest.mark.parametrize("nants", [3, 19, 54, 91, 150, 200])
def test_omnical_float64_layouts(nants):
    from hera_gpu_gb300 import omnical
    from oracle import omnical_oracle
    ggu, nubls = synth.hex_redundant_layout(nants)
    g0, u0, d, w = synth.redundant_data(ggu, nubls, 3, seed=nants, noise=0.05)
    w = np.where(np.random.default_rng(nants).random(w.shape) < 0.05, 0.0, w)
    a = [x.astype(t) for x, t in ((g0, np.complex128), (u0, np.complex128), (d, np.complex128),
                                  (w, np.float64))]
    got = omnical(ggu, *a, 1e-10, 12, precision=2)
    ref = omnical_oracle(ggu, *a, 1e-10, 12, precision=2)
    for x in ("gains", "ubls"):  # (a unique baseline may be flagged altogether)
        finite = np.isfinite(ref[x])
        np.testing.assert_array_equal(np.isfinite(got[x]), finite)
        assert (np.abs(got[x] - ref[x])[finite].max(initial=0)
                <= 1e-11 * np.abs(ref[x][finite]).max(initial=1))
    np.testing.assert_array_equal(got["iters"], ref["iters"])


# a float64 problem gives the same bits in a call of many problems (CTAs of 256
# threads) as alone (up to 512)
@gpu
@pytest.mark.parametrize("nants", [37, 54, 70])
def test_omnical_float64_alone_and_among_many(nants):
    from hera_gpu_gb300 import omnical
    ggu, nubls = synth.hex_redundant_layout(nants)
    a = [np.concatenate([x] * 110) for x in
         synth.redundant_data(ggu, nubls, 3, seed=nants, noise=0.05)]
    many = omnical(ggu, *[x.astype(t) for x, t in zip(a, (np.complex128, np.complex128,
                                                          np.complex128, np.float64))],
                   1e-10, 12, precision=2)
    one = omnical(ggu, *[x[:3].astype(t) for x, t in zip(a, (np.complex128, np.complex128,
                                                             np.complex128, np.float64))],
                  1e-10, 12, precision=2)
    for x in ("gains", "ubls", "chisq", "iters", "conv"):
        np.testing.assert_array_equal(many[x][-3:], one[x])
        np.testing.assert_array_equal(many[x][:3], one[x])


# antenna blocks of the fused forms (32, 64, 96 and 128 rows; one to five
# blocks), at their edges
@gpu
@pytest.mark.parametrize("method", ["tc", "tc_fp16"])
@pytest.mark.parametrize("nant", [31, 32, 33, 64, 65, 96, 97, 128, 129, 161, 192, 193, 257, 288,
                                  289, 385, 520, 641])
def test_antenna_blocks(nant, method):
    args = sim(nant, 700, ntimes=2, seed=nant)
    v = vis_gpu(*args, precision=1, method=method)
    check_hermitian(v)
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
    assert rel_frobenius(v, ref).max() <= 1e-4
    if method == "tc":
        # every entry on the scale of its antennas' powers (split BF16 operands
        # carry 16 bits): a misplaced block or a sign of one pair would be of
        # order 1
        p = np.sqrt(np.einsum("taa->ta", ref.real))
        assert np.abs(v - ref).max() <= 1e-4 * (p[:, :, None] * p[:, None, :]).max()


# calls that leave CTAs or clusters idle at the shortest regular chunk take
# shorter ones: one source, one chunk, a last chunk of a few sources
@gpu
@pytest.mark.parametrize("method", ["tc", "tc_fp16"])
@pytest.mark.parametrize("nant,nsrc,ntimes", [(16, 1, 1), (16, 130, 1), (40, 2047, 7), (200, 257, 1),
                                              (200, 20000, 1), (350, 3001, 5), (641, 4099, 2)])
def test_small_call_chunks(nant, nsrc, ntimes, method):
    args = sim(nant, nsrc, ntimes=ntimes, seed=nsrc)
    v = vis_gpu(*args, precision=1, method=method)
    check_hermitian(v)
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
    up = np.abs(ref).max(axis=(1, 2)) > 0
    assert rel_frobenius(v[up], ref[up]).max(initial=0) <= 1e-4
    assert not v[~up].any()


# order of the records: by counting (one pixel, a few, a box of hundreds) and
# by sorting (a box beyond 512 pixels); blocks of 1024 sources that form the
# counts before them (up to 4096 sources) and that read them.  A lost or
# doubled source is of order 1 / sqrt(nsrc) >= 1e-2, far above the tolerance
@gpu
@pytest.mark.parametrize("P", [2, 15, 63, 301])
@pytest.mark.parametrize("nsrc", [31, 1023, 1025, 4096, 4097, 8193])
def test_record_order(nsrc, P):
    args = sim(4, nsrc, ntimes=2, P=P, seed=nsrc + P)
    v = vis_gpu(*args, precision=1, method="tc")
    check_hermitian(v)
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in args])
    assert rel_frobenius(v, ref).max() <= 1e-4


# host calls around the limits of page-locked staging (512 KB of inputs, 64 KB
# of output: 90 antennas), small and large ones in turn through one context
@gpu
def test_host_calls_staged_and_not():
    cases = [sim(nant, nsrc, seed=nsrc) for nant, nsrc in
             [(90, 1000), (91, 27000), (90, 26000), (91, 1000), (8, 40000), (8, 1)]]
    first = [vis_gpu(*a, precision=1, method="tc") for a in cases]
    for a, v in zip(cases, first):
        ref = vis_oracle(*[x.astype(np.float64) if isinstance(x, np.ndarray) else x for x in a])
        if ref.any():
            assert rel_frobenius(v, ref).max() <= 1e-4
    for a, v in zip(cases[::-1], first[::-1]):
        np.testing.assert_array_equal(vis_gpu(*a, precision=1, method="tc"), v)


# chunks of several accumulator runs: a last chunk of one run and less, chunks
# beyond the sources above the horizon
@gpu
@pytest.mark.parametrize("method", ["tc", "tc_fp16"])
@pytest.mark.parametrize("nant,nsrc,ntimes", [(33, 20000, 60), (70, 6100, 200), (260, 9000, 40)])
def test_chunks_of_several_runs(nant, nsrc, ntimes, method):
    args = sim(nant, nsrc, ntimes=ntimes, seed=nant)
    v = vis_gpu(*args, precision=1, method=method)
    check_hermitian(v)
    t = [0, ntimes // 2, ntimes - 1]
    part = (args[0], args[1], args[2][t], *args[3:])
    ref = vis_oracle(*[a.astype(np.float64) if isinstance(a, np.ndarray) else a for a in part])
    assert rel_frobenius(v[t], ref).max() <= 1e-4
