"""The bit-packed step's kernels at the sides where one takes over from another
(one CTA, several CTAs with blocked generations, tiles, band walk) and where a row
ends inside, at or after a word; square and rectangular, one generation and
several per call (odd and even counts leave the grid in different frames), and
under stream capture.  Bit-exact against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.test_packed_walk import rows_cols_step

pytestmark = pytest.mark.gpu


def rule_of(r):
    N = (2 * r + 1) ** 2
    return (N // 3, N // 2, int(0.4 * N), int(0.46 * N))


@pytest.mark.parametrize("radius", [1, 2, 5, 8, 12, 16, 17])
def test_sides_vs_oracle(radius):
    import cat_cpu_b200 as C
    rng = np.random.default_rng(radius)
    rule = rule_of(radius)
    for n in (40, 63, 64, 65, 90, 91, 127, 128, 129, 300, 1000, 1024, 1025, 1057, 2111):
        g = (rng.random((n, n)) < 0.45).astype(np.uint8)
        with C.CUDASolver(n, radius, rule, variant=C.VARIANT_PACKED) as s:
            s.setState(g)
            for steps in (1, 2, 7, 12) if n < 2000 else (3,):
                s.doSteps(steps)
                g = O.run(g, radius, rule, steps)
                assert np.array_equal(s.getCurrentState(), g), (n, radius, steps)
            s.synchronize()


@pytest.mark.parametrize("rows,n,radius", [(17, 96, 16), (5, 1024, 5), (8, 40, 8), (700, 64, 3), (33, 1500, 4), (1200, 50, 2)])
def test_rectangles_vs_numpy(rows, n, radius):
    import cat_cpu_b200 as C
    rng = np.random.default_rng(rows)
    rule = rule_of(radius)
    g = (rng.random((rows, n)) < 0.45).astype(np.uint8)
    with C.CUDASolver(n, radius, rule, variant=C.VARIANT_PACKED, rows=rows) as s:
        s.setState(g)
        for steps in (1, 6):
            s.doSteps(steps)
            for _ in range(steps):
                g = rows_cols_step(g, radius, rule)
            assert np.array_equal(s.getCurrentState(), g), (rows, n, radius, steps)


@pytest.mark.parametrize("n,radius", [(64, 5), (300, 5), (2048, 8), (6500, 1)])
def test_captured_steps_replay(n, radius):
    """An even number of generations captured into a caller's graph advances the
    grid on every replay."""
    import torch
    import cat_cpu_b200 as C
    rule = rule_of(radius)
    g = (np.random.default_rng(n).random((n, n)) < 0.45).astype(np.uint8)
    stream = torch.cuda.Stream()
    with C.CUDASolver(n, radius, rule, variant=C.VARIANT_PACKED) as s:
        s.set_stream(stream.cuda_stream)
        s.setState(g)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            s.doSteps(4)
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.getCurrentState(), O.run(g, radius, rule, 8))
        del graph


@pytest.mark.parametrize("n,radius", [(64, 1), (100, 5), (1000, 12), (300, 28), (300, 29)])
def test_auto_names_plain_and_takes_its_parameters(n, radius):
    """The default solver: same info, parameters and results on either side of the
    radius where it changes kernels."""
    import cat_cpu_b200 as C
    rule = rule_of(radius)
    g = (np.random.default_rng(n + radius).random((n, n)) < 0.45).astype(np.uint8)
    with C.CUDASolver(n, radius, rule) as s, C.CUDASolver(n, radius, rule, variant=C.VARIANT_PLAIN) as p:
        for field in ("variant", "halo", "pitch", "temporal_depth", "operand_bits", "radius", "n", "rows"):
            assert getattr(s.info, field) == getattr(p.info, field), field
        for solver in (s, p):
            solver.set_param("band_rows", 32)
            if radius <= 5:
                solver.set_param("depth", 2)
                assert solver.info.temporal_depth == 2
            else:
                with pytest.raises(C.LtlError):
                    solver.set_param("depth", 2)
            with pytest.raises(C.LtlError):
                solver.set_param("wait_limit_ns", 10**9)
            solver.setState(g)
            solver.doSteps(5)
            assert np.array_equal(solver.getCurrentState(), O.run(g, radius, rule, 5))
            assert solver.population() == int(O.run(g, radius, rule, 5).sum())


@pytest.mark.parametrize("n,radius", [(12001, 1), (12032, 2), (14001, 4), (20033, 5), (20032, 1)])
def test_short_bands_vs_long_bands_and_plain(n, radius):
    """Grids large enough for the band walk's short bands (within the L2, and with
    frames that do not fit it): the same cells as with long bands and as the plain
    solver's, which counts in another way."""
    import torch
    import cat_cpu_b200 as C
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    g = (torch.rand((n, n), generator=gen, device="cuda") < 0.45).to(torch.uint8)
    torch.cuda.synchronize()
    got = []
    for variant, band_rows in ((C.VARIANT_PACKED, 0), (C.VARIANT_PACKED, 500), (C.VARIANT_PLAIN, 0)):
        out = torch.empty_like(g)
        torch.cuda.synchronize()
        with C.CUDASolver(n, radius, rule_of(radius), variant=variant) as s:
            if band_rows:
                s.set_param("band_rows", band_rows)
            s.upload_device(g.data_ptr(), n)
            s.doSteps(3)
            s.download_device(out.data_ptr(), n)
            s.synchronize()
        got.append(out)
    assert int(got[0].sum()) > 0
    assert torch.equal(got[0], got[1])
    assert torch.equal(got[0], got[2])


@pytest.mark.parametrize("variant,n,radius,steps", [(-1, 700, 17, 10), (-1, 7000, 5, 14), (0, 1000, 5, 22), (0, 300, 1, 23),
                                                    (1, 5200, 5, 16), (2, 700, 20, 8)])
def test_captured_steps_of_many_passes(variant, n, radius, steps):
    """As many passes in one captured call as the solver otherwise replays from a
    graph of its own, also where it has made that graph before."""
    import torch
    import cat_cpu_b200 as C
    rule = rule_of(radius)
    g = (np.random.default_rng(n).random((n, n)) < 0.45).astype(np.uint8)
    stream = torch.cuda.Stream()
    with C.CUDASolver(n, radius, rule, variant=variant) as s, C.CUDASolver(n, radius, rule, variant=0) as one:
        one.set_param("depth", 1)
        one.setState(g)
        one.doSteps(2 * steps)
        want = one.getCurrentState()
        s.set_stream(stream.cuda_stream)
        for before in (0, 48):
            s.doSteps(before)
            s.setState(g)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                s.doSteps(steps)
                s.doSteps(steps)
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(s.getCurrentState(), want), before
            del graph


@pytest.mark.parametrize("n,radius", [(200, 12), (1000, 12), (1000, 16), (3001, 8)])
def test_changes_between_the_walk_and_the_runs(n, radius):
    """A set band height keeps a small grid on the band walk, 0 gives it back."""
    import cat_cpu_b200 as C
    rule = rule_of(radius)
    g = (np.random.default_rng(n).random((n, n)) < 0.45).astype(np.uint8)
    with C.CUDASolver(n, radius, rule, variant=C.VARIANT_PACKED) as s:
        s.setState(g)
        for band in (0, 64, 0, 100):
            s.set_param("band_rows", band)
            s.doSteps(9)
            g = O.run(g, radius, rule, 9)
            assert np.array_equal(s.getCurrentState(), g), (n, radius, band)


@pytest.mark.parametrize("rows,n,radius", [(13000, 15001, 19), (14001, 14001, 28), (19616, 19616, 20), (19616, 19616, 28),
                                           (1500000, 60, 19)])
def test_large_grids_without_the_ring_vs_plain(rows, n, radius):
    """Radii whose ring leaves one CTA per SM, where grids are too large for that; and rows
    of fewer than 64 cells, which keep it."""
    import torch
    import cat_cpu_b200 as C
    N = (2 * radius + 1) ** 2
    rule = (int(0.45 * N), N, int(0.45 * N), N)  # above the mean count: domains of both kinds
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    g = (torch.rand((rows, n), generator=gen, device="cuda") < 0.45).to(torch.uint8)
    torch.cuda.synchronize()
    got = []
    for variant in (C.VARIANT_PACKED, C.VARIANT_PLAIN):
        out = torch.empty_like(g)
        torch.cuda.synchronize()
        with C.CUDASolver(n, radius, rule, variant=variant, rows=rows) as s:
            s.upload_device(g.data_ptr(), n)
            s.doSteps(9)
            s.download_device(out.data_ptr(), n)
            s.synchronize()
        got.append(out)
    assert 0 < int(got[0].sum()) < rows * n
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("n,radius", [(2016, 23), (2016, 24), (2048, 24), (2048, 28), (2080, 29), (2049, 28)])
def test_default_solver_where_it_changes_kernels(n, radius):
    import cat_cpu_b200 as C
    rule = rule_of(radius)
    g = (np.random.default_rng(n + radius).random((n, n)) < 0.45).astype(np.uint8)
    with C.CUDASolver(n, radius, rule) as s, C.CUDASolver(n, radius, rule, variant=C.VARIANT_PLAIN) as p:
        for solver in (s, p):
            solver.setState(g)
            solver.doSteps(2)
        assert np.array_equal(s.getCurrentState(), p.getCurrentState())
        assert s.info.variant == p.info.variant == C.VARIANT_PLAIN
        assert s.population() == p.population() > 0
