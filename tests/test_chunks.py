"""The split of the fused kernel's sources and antennas, from the library's own
host code (fake_gpu.py)."""
import ctypes
import os
import random
import sys

import pytest

import fake_gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

SMS = 152


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    g = fake_gpu.FakeGpu(fake_gpu.build_library(tmp_path_factory.mktemp("fake")), 1 << 30)
    yield g.lib
    g.close()


def chunk_and_run(lib, nsrc, ntimes, nfreq, nant, form=0, spread=True):
    run = ctypes.c_int()
    chunk = lib._ZN2hv16tc_chunk_sourcesEiiiiiibPi(
        nsrc, ntimes, nfreq, lib._ZN2hv13tc_num_groupsEi(nant),
        lib._ZN2hv13tc_block_rowsEii(nant, form), SMS, ctypes.c_bool(spread), ctypes.byref(run))
    return chunk, run.value


def shapes(n):
    rng = random.Random(1)
    for _ in range(n):
        yield (int(1000 * 2 ** rng.uniform(0, 10.04)), rng.randint(1, 60), rng.randint(1, 8),
               rng.randint(1, 512))


# the tensor core's accumulation loses in proportion to the sources it sums at a
# time: about 40 spans a CTA or cluster, each in whole flushes of 2048 and a rest,
# set how many that are on average
def test_accumulator_runs_are_no_longer_than_flushes_of_spans(lib):
    for nsrc, ntimes, nfreq, nant in shapes(3000):
        up, n = max(nsrc // 2, 1), ntimes * nfreq * lib._ZN2hv13tc_num_groupsEi(nant)
        span = min(32768, max(1024, -(-up // max(1, -(-40 * SMS // n)))))
        span = -(-span // 32) * 32
        pieces = [min(2048, k) for s in range(0, up, span)
                  for k in range(min(span, up - s), 0, -2048)]
        chunk, run = chunk_and_run(lib, nsrc, ntimes, nfreq, nant)
        assert run % 32 == 0 and chunk % run == 0
        runs = [min(run, up - s) for s in range(0, up, run)]
        mean = [sum(k * k for k in x) / up for x in (pieces, runs)]
        assert mean[1] <= 1.03 * mean[0], (nsrc, ntimes, nfreq, nant)


# the benchmark's account of the issued MMAs restates both
@pytest.mark.parametrize("method,form", [("tc", 0), ("tc_fp16", 1)])
def test_the_benchmark_restates_the_split(lib, method, form):
    for nsrc, ntimes, nfreq, nant in shapes(1000):
        assert bench.tc_num_groups(nant, method) == lib._ZN2hv13tc_num_groupsEi(nant)
        assert bench.tc_block_rows(nant, method) == lib._ZN2hv13tc_block_rowsEii(nant, form)
        got = bench.tc_chunk(nsrc, ntimes * nfreq, nant, method, SMS)
        assert got == chunk_and_run(lib, nsrc, ntimes, nfreq, nant, form, spread=False)[0]
