"""Precision 2 where antennas are bright on different sources: each entry of V
is held to the FP64 sum's own bound, relative to sum_s |v_a| |v_b|."""
import numpy as np
import pytest

from hera_gpu_gb300 import synth, vis_gpu
from oracle import vis_oracle

gpu = pytest.mark.gpu
C = 299792458.0


def split_sim(nant, nsrc, faint, seed, odd=slice(1, None, 2)):
    """Antennas `odd` see the west with 1 and the east with `faint`, the others
    the reverse; no source near the border of the two halves."""
    c = synth.config_array(seed=seed, nant=nant, nsrc=nsrc, ntimes=1, P=15)
    east = (c["eq2tops"][0] @ c["crd_eq"])[0]
    keep = np.abs(east) > 0.3              # the border: pixels 6 and 8 of 15, |l| <= 1/7
    bm = np.ones((nant, 15, 15))
    bm[:, :, 7:] = faint
    bm[odd] = 1.0
    bm[odd, :, :8] = faint
    return (c["antpos"], float(c["freqs"][0]), c["eq2tops"],
            np.ascontiguousarray(c["crd_eq"][:, keep]), c["I_sky"][keep], bm)


def entry_bound(args):
    """sum_s |v_a| |v_b| (the beams are not negative: the sum without phases)
    times the rounding of an FP64 sum of n products (2 n 2^-53), of the
    amplitudes (16) and of U and the phases (8 roundings of the largest |U| in
    cycles), once for each side of the comparison."""
    dark = vis_oracle(args[0] * 0.0, *args[1:])
    cycles = np.sqrt((args[0] ** 2).sum(axis=1)).max() * args[1] / C
    n = args[3].shape[1]
    return 2 * (2 * n + 16 + 2 * np.pi * 8 * cycles) * 2.0 ** -53 * dark.real


# one and two antenna blocks; one source window; a beam of zeros on the dark half
@gpu
@pytest.mark.parametrize("nant,nsrc", [(2, 300), (35, 900), (150, 500)])
@pytest.mark.parametrize("faint", [1e-3, 1e-6, 1e-10, 1e-30, 0.0])
def test_antennas_bright_on_different_sources(nant, nsrc, faint):
    args = split_sim(nant, nsrc, faint, seed=nant)
    v = vis_gpu(*args, precision=2)
    assert np.all(np.abs(v - vis_oracle(*args)) <= entry_bound(args))


# one such antenna, in the last antenna block, and in one of two times only
@gpu
def test_one_antenna_and_one_time():
    args = list(split_sim(140, 700, 1e-8, seed=5, odd=slice(139, 140)))
    quarter = np.array([[0.0, 1.0, 0.0], [-1.0, 0.0, 0.0], [0.0, 0.0, 1.0]])
    args[2] = np.stack([args[2][0], quarter @ args[2][0]])
    v = vis_gpu(*args, precision=2)
    assert np.all(np.abs(v - vis_oracle(*args)) <= entry_bound(args))


# the window of sources that holds them decides, also beyond the first 65536
@gpu
def test_bright_sources_in_the_second_window():
    args = list(split_sim(3, 150_000, 1e-9, seed=6))
    # the catalogue's last sources alone are bright
    args[4] = np.where(np.arange(len(args[4])) < 0.97 * len(args[4]), 1e-18, 1.0) * args[4]
    v = vis_gpu(*args, precision=2)
    assert np.all(np.abs(v - vis_oracle(*args)) <= entry_bound(args))


# ordinary beams keep the digit form: with an antenna that sees only what the
# others do not, the slice takes the SIMT product, whose bits differ
@gpu
@pytest.mark.parametrize("beams", ["airy", "random"])
def test_ordinary_beams_keep_the_digit_form(beams):
    c = synth.config_array(seed=9, nant=200, nsrc=2000, ntimes=1, P=31)
    bm = synth.beams_for(c, dtype=np.float64)[0]
    if beams == "random":
        bm = np.random.default_rng(1).random(bm.shape)
    args = [c["antpos"], float(c["freqs"][0]), c["eq2tops"], c["crd_eq"], c["I_sky"], bm]
    v = vis_gpu(*args, precision=2)
    assert np.all(np.abs(v - vis_oracle(*args)) <= entry_bound(args))
    bm[:, :, 24:] = 0.0                    # the east is dark, but for one antenna more
    v = vis_gpu(*args, precision=2)
    east = np.zeros((1, 31, 31))
    east[:, :, 26:] = 1.0
    other = vis_gpu(np.concatenate([args[0], args[0][:1]]), *args[1:5],
                    np.concatenate([bm, east]), precision=2)[:, :200, :200]
    assert np.any(other != v)
    assert np.all(np.abs(other - v) <= entry_bound(args))
