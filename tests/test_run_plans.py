"""The host-side plans of launches whose CTAs wait for one another, compiled from the
kernels' own headers: a batch's groups of CTAs all fit on the chip at once, and the
blocks of a small grid's generations add up and end in the right frame."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plans") / "plans.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "cat_cpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "batch_split_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def split(host, grids, ctas, per_sm):
    n, r = (np.array(v, dtype=np.int32) for v in zip(*grids))
    sizes = np.zeros(len(grids), dtype=np.int32)
    times, alone = np.zeros(len(grids)), np.zeros(len(grids))
    p = [v.ctypes.data_as(ctypes.c_void_p) for v in (n, r)]
    host.batch_split_host(*p, len(grids), ctas, per_sm, *[v.ctypes.data_as(ctypes.c_void_p) for v in (sizes, times, alone)])
    return sizes, times, alone


def ensembles():
    rng = np.random.default_rng(6)
    yield [(4096, 5)]
    yield [(20000, 2)]
    yield [(16, 5)]
    yield [(64, 1)] * 8
    yield [(2000, 8)] + [(64, 1)] * 500
    yield [(300000, 16), (16, 16)]
    for count, lo, hi, rmax in ((7, 16, 40, 16), (64, 64, 2048, 8), (1024, 64, 2048, 8), (20, 40, 3000, 16), (3000, 64, 128, 2)):
        side = np.exp(rng.uniform(np.log(lo), np.log(hi), count)).astype(int)
        yield [(int(n), int(rng.integers(1, rmax + 1))) for n in side]


@pytest.mark.parametrize("per_sm", [1, 2, 4])
def test_groups_fit_the_chip_and_pay(host, per_sm):
    ctas = 148 * per_sm
    for grids in ensembles():
        sizes, times, alone = split(host, grids, ctas, per_sm)
        assert (sizes >= 1).all()
        assert sizes[sizes > 1].sum() <= ctas, grids[:3]
        # a group is made only where the model has it faster than one CTA
        assert (times[sizes > 1] < alone[sizes > 1]).all(), grids[:3]
        # and the work adds up to no more than one CTA per grid takes on as many CTAs
        assert (sizes * times).sum() / ctas <= max(alone.sum() / ctas, alone.max()) * 1.05


def test_a_large_grid_gets_the_chip(host):
    sizes, _, _ = split(host, [(4096, 5)], 592, 4)
    assert sizes[0] > 100
    sizes, _, _ = split(host, [(64, 1)] * 5000, 592, 4)
    assert (sizes == 1).all()


def test_blocks_of_generations(host):
    gens = (ctypes.c_int * 1024)()
    for steps in list(range(1, 70)) + [255, 256, 511, 512]:
        for depth in range(1, 13):
            blocks = host.run_blocks_host(steps, min(depth, steps), gens)
            got = list(gens[:blocks])
            assert sum(got) == steps and min(got) >= 1, (steps, depth, got)
            assert blocks % 2 == steps % 2, (steps, depth)
            # the launch sizes its shared memory for the first block
            assert max(got) == got[0] <= depth, (steps, depth, got)
