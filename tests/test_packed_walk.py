"""The bit-packed band walk, compiled for the host from the kernels' own header
(cat_cpu_b200/csrc/packed_core.cuh) and run lane by lane: every form of it (one
or two words per lane, whole, ragged and tiny rows, with and without the ring of
window counts) against the oracle, with every read checked to lie inside the
grid; and its interval rule against the scalar one for every count."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("walk") / "walk.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "cat_cpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "packed_walk_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def words_of(grid, wp, rng):
    rows, n = grid.shape
    nw = (n + 31) // 32
    padded = np.zeros((rows, nw * 32), dtype=np.uint8)
    padded[:, :n] = grid
    past = nw * 32 - n  # bits past n: the row's first cells from 64 cells on, else anything
    padded[:, n:] = grid[:, :past] if n >= 64 else rng.integers(0, 2, size=(rows, past))
    out = rng.integers(0, 2**32, size=(rows, wp), dtype=np.uint32)
    out[:, :nw] = np.packbits(padded, axis=1, bitorder="little").view("<u4")
    return out


def cells_of(words, n):
    return np.unpackbits(np.ascontiguousarray(words).view(np.uint8), axis=1, bitorder="little")[:, :n]


def rows_cols_step(grid, r, rule):
    """One generation of a rows x n torus (the oracle's step is for squares)."""
    smin, smax, bmin, bmax = rule
    k = np.zeros(grid.shape, dtype=np.int64)
    for d in range(-r, r + 1):
        k += np.roll(grid, d, axis=0)
    box = sum(np.roll(k, d, axis=1) for d in range(-r, r + 1)) - grid
    return np.where(grid > 0, (box >= smin) & (box <= smax), (box >= bmin) & (box <= bmax)).astype(np.uint8)


def check(host, grid, want, r, rule, words, ring, band, rng):
    rows, n = grid.shape
    wp = (((n + 31) // 32) + 3) // 4 * 4
    cur = words_of(grid, wp, rng)
    nxt = np.zeros_like(cur)
    rc = host.packed_step_host(cur.ctypes.data_as(ctypes.c_void_p), nxt.ctypes.data_as(ctypes.c_void_p), wp, n, rows, r,
                               *rule, words, ring, band)
    if rc == 1:
        return 0
    assert rc == 0, (n, rows, r, words, ring, band, rc)
    assert np.array_equal(cells_of(nxt, n), want), (n, rows, r, words, ring, band)
    if n >= 64:  # the step keeps the rows joined
        nw = (n + 31) // 32
        assert np.array_equal(cells_of(nxt, 32 * nw)[:, n:], want[:, :32 * nw - n]), (n, rows, r, words, ring, band)
    return 1


@pytest.mark.parametrize("radius", [1, 2, 3, 4, 5, 7, 8, 11, 14, 16, 17, 24, 32])
def test_walk_vs_oracle(host, radius):
    rng = np.random.default_rng(radius)
    N = (2 * radius + 1) ** 2
    ran = 0
    sides = [radius, radius + 1, 31, 32, 33, 47, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 191, 224]
    for n in sorted({s for s in sides if s >= radius}):
        grid = (rng.random((n, n)) < 0.45).astype(np.uint8)
        lo = int(rng.integers(0, N // 2))
        rule = (lo, lo + N // 3, int(0.4 * N), int(0.46 * N))
        want = O.step(grid, radius, rule)
        for words in (1, 2):
            for ring in (0, 1):
                ran += check(host, grid, want, radius, rule, words, ring, int(rng.integers(1, n + 3)), rng)
    assert ran >= 20


@pytest.mark.parametrize("radius", [1, 2, 3, 5, 8, 11, 16])
def test_tiles_vs_oracle(host, radius):
    """Tiles that do and do not divide the grid, narrow and full ones."""
    rng = np.random.default_rng(40 + radius)
    N = (2 * radius + 1) ** 2
    for n in sorted({s for s in (radius, 17, 33, 64, 65, 96, 97, 160, 257, 1100) if s >= radius}):
        rows = n if n < 300 else 40
        grid = (rng.random((rows, n)) < 0.45).astype(np.uint8)
        rule = (N // 3, N // 2, int(0.4 * N), int(0.46 * N))
        want = rows_cols_step(grid, radius, rule)
        nw = (n + 31) // 32
        wp = (nw + 3) // 4 * 4
        for tr, tc, threads, band in ((rows, min(nw, 32), 96, 5), (7, max(1, nw // 2), 64, 2), (1, min(nw, 32), 32, 1)):
            cur = words_of(grid, wp, rng)
            nxt = np.zeros_like(cur)
            tc = min(tc, 32)
            rc = host.packed_tiles_host(cur.ctypes.data_as(ctypes.c_void_p), nxt.ctypes.data_as(ctypes.c_void_p), wp, n,
                                        rows, radius, *rule, tr, tc, threads, band)
            assert rc == 0 and np.array_equal(cells_of(nxt, n), want), (n, rows, radius, tr, tc, rc)
            if n >= 64:
                assert np.array_equal(cells_of(nxt, 32 * nw)[:, n:], want[:, :32 * nw - n]), (n, rows, radius, tr, tc)


def test_walk_on_strips(host):
    rng = np.random.default_rng(5)
    for rows, n, r in ((8, 200, 8), (9, 64, 5), (40, 130, 3), (300, 40, 5), (17, 96, 16)):
        grid = (rng.random((rows, n)) < 0.45).astype(np.uint8)
        N = (2 * r + 1) ** 2
        rule = (N // 3, N // 2, int(0.4 * N), int(0.46 * N))
        for words in (1, 2):
            check(host, grid, rows_cols_step(grid, r, rule), r, rule, words, 1, 7, rng)


@pytest.mark.parametrize("radius", [1, 2, 5, 16, 32])
def test_rule_every_count(host, radius):
    """Intervals inside, outside and across the counts' range, empty ones, the whole range."""
    N = (2 * radius + 1) ** 2
    big = 2**31 - 1
    ends = [-big, -1, 0, 1, N // 3, N // 2, N - 1, N, N + 1, big]
    rng = np.random.default_rng(radius)
    counts = range(N + 1) if N < 200 else sorted({0, 1, 2, N - 2, N - 1, N, N // 2 - 1, N // 2, N // 2 + 1, N // 3 - 1,
                                                  N // 3, N // 3 + 1} | set(rng.integers(0, N, 30).tolist()))
    for _ in range(120):
        smin, smax, bmin, bmax = (int(v) for v in rng.choice(ends, 4))
        for B in counts:
            if B < N:
                assert packed(host, radius, smin, smax, bmin, bmax, B, 0) == (bmin <= B <= bmax), (smin, smax, bmin, bmax, B)
            if B > 0:
                assert packed(host, radius, smin, smax, bmin, bmax, B, 1) == (smin <= B - 1 <= smax), (smin, smax, bmin, bmax, B)


def packed(host, *args):
    return host.packed_rule_host(*args)
