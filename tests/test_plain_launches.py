"""The plain form's launches: few slices at a time as well as many."""
import numpy as np
import pytest

import fake_gpu
from hera_gpu_gb300 import synth, vis_gpu, vis_gpu_multifreq

gpu = pytest.mark.gpu


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    g = fake_gpu.FakeGpu(fake_gpu.build_library(tmp_path_factory.mktemp("fake")), 64 << 30)
    yield g
    g.close()


def blocks(log, name):
    return [b for op, _, b in log if op.startswith("launch ") and name in op]


# a launch of few sources gives a warp one of them instead of 64 in a row: as many
# warps (8 a block) as there are sources and groups of 32 antennas
@pytest.mark.parametrize("nant,nsrc,ntimes", [(1, 100, 1), (4, 100, 1), (300, 100, 1), (16, 1000, 4),
                                              (350, 1000, 1)])
def test_phasors_of_few_sources(fake, nant, nsrc, ntimes):
    assert fake.call(fake.context(), 1, "plain", nant, nsrc, ntimes) == 0
    groups = -(-nant // 128) * 4
    assert 8 * sum(blocks(fake.log(), "gen_phasors")) >= nsrc * groups * ntimes


def test_phasors_of_many_sources(fake):
    assert fake.call(fake.context(), 1, "plain", 350, 100_000, 5) == 0
    assert 8 * sum(blocks(fake.log(), "gen_phasors")) <= 1.01 * 100_000 / 64 * 12 * 5


# blocks that are on the SMs at once (two each) take the kernel that ends sooner
@pytest.mark.parametrize("nant,nsrc,ntimes,few", [
    (16, 1000, 1, True), (350, 20_000, 1, True), (350, 20_000, 4, True), (350, 100_000, 1, True),
    (350, 100_000, 2, True), (350, 100_000, 5, False), (700, 5000, 5, False), (512, 8000, 8, True)])
def test_products_of_few_blocks(fake, nant, nsrc, ntimes, few):
    assert fake.call(fake.context(), 1, "plain", nant, nsrc, ntimes) == 0
    log = fake.log()
    assert bool(blocks(log, "herk_tile_kernel")) == few
    assert bool(blocks(log, "herk_plain_kernel")) != few


# both kernels and every span give the same bits: a call of many slices and its
# single slices; a chunk of 4096 sources and a rest, stages of 16 and a rest
@gpu
@pytest.mark.parametrize("nant,nsrc", [(5, 9001), (130, 9001), (70, 300)])
def test_slices_give_the_same_bits_together_and_alone(nant, nsrc):
    c = synth.config_array(seed=nant, nant=nant, nsrc=nsrc, ntimes=60, nfreq=4, fmin=1e8, fmax=2e8, P=9)
    bm = synth.beams_for(c, dtype=np.float32)
    a = [c["antpos"], c["eq2tops"], c["crd_eq"], c["I_sky"]]
    a = [x.astype(np.float32) for x in a]
    many = vis_gpu_multifreq(a[0], c["freqs"], *a[1:], bm, precision=1, method="plain")
    for f, t in ((0, 0), (1, 17), (3, 59)):
        one = vis_gpu(a[0], float(c["freqs"][f]), a[1][t:t + 1], *a[2:], bm[f], precision=1,
                      method="plain")
        np.testing.assert_array_equal(one[0], many[f, t])
