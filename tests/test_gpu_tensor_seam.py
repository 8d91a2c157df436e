"""The tensor step where the row's end lies inside a word: sides around the smallest
that stage words through shared memory, in every operand mode; rows of tiles whose
last tile is full, partial, or ends next to the seam.  Bit-exact against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [1, 5, 6, 16, 17, 33, 60, 91, 113, 128])
def test_ragged_sides_vs_oracle(radius):
    import cat_cpu_b200 as C
    rng = np.random.default_rng(radius)
    N = (2 * radius + 1) ** 2
    rule = (N // 3, N // 2, int(0.4 * N), int(0.46 * N))
    nb = 1 if radius <= 32 else (128 + 2 * radius + 127) // 128
    low = 128 * nb + radius
    for n in sorted({low - 1, low, low + 1, 383, 385, 511, 513, 640 + 17, 1000, 1025}):
        if n < radius:
            continue
        g = (rng.random((n, n)) < 0.45).astype(np.uint8)
        with C.CUDASolver(n, radius, rule, variant=C.VARIANT_TENSOR) as s:
            s.setState(g)
            for steps in (2, 1, 5):  # many generations per launch, and one
                s.doSteps(steps)
                s.synchronize()
                g = O.run(g, radius, rule, steps)
                assert np.array_equal(s.getCurrentState(), g), (n, radius, steps)


def test_timeout_in_a_launch_of_many_generations():
    """A withheld completion signal in one CTA: the others wait for its generation in
    vain, every wait is bounded, the host sees LTL_ETIMEOUT, and the solver works on."""
    import cat_cpu_b200 as C
    n, r = 700, 5
    g = (np.random.default_rng(1).random((n, n)) < 0.45).astype(np.uint8)
    with C.CUDASolver(n, r, O.BOSCO_R5, variant=C.VARIANT_TENSOR) as s:
        s.set_param("wait_limit_ns", 20_000_000)
        s.set_param("inject_missing_commit", 1)
        s.setState(g)
        s.doSteps(4)
        with pytest.raises(C.LtlError) as e:
            s.synchronize()
        assert e.value.code == C.ltl.ETIMEOUT
        s.set_param("inject_missing_commit", 0)
        s.setState(g)
        s.doSteps(6)
        s.synchronize()
        assert np.array_equal(s.getCurrentState(), O.run(g, r, O.BOSCO_R5, 6))


def test_captured_generations_replay():
    import torch
    import cat_cpu_b200 as C
    n, r = 500, 6
    rule = O.scaled_rule(r)
    g = (np.random.default_rng(2).random((n, n)) < 0.45).astype(np.uint8)
    stream = torch.cuda.Stream()
    with C.CUDASolver(n, r, rule, variant=C.VARIANT_TENSOR) as s:
        s.set_stream(stream.cuda_stream)
        s.setState(g)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            s.doSteps(4)
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(s.getCurrentState(), O.run(g, r, rule, 8))
        del graph


def test_solvers_of_large_and_small_shared_memory():
    """Radii that share a kernel and differ in the shared memory they launch it with, made
    in falling order of that and stepped afterwards."""
    import cat_cpu_b200 as C
    rng = np.random.default_rng(7)
    made = []
    for n, r in ((700, 48), (700, 33), (700, 17), (700, 127), (700, 113), (512, 90), (300, 90), (640, 32), (500, 80), (500, 49)):
        N = (2 * r + 1) ** 2
        rule = (N // 3, N // 2, int(0.4 * N), int(0.46 * N))
        s = C.CUDASolver(n, r, rule, variant=C.VARIANT_TENSOR)
        g = (rng.random((n, n)) < 0.45).astype(np.uint8)
        s.setState(g)
        made.append((s, n, r, rule, g))
    for s, n, r, rule, g in made:
        s.doSteps(3)
        s.doSteps(1)
        s.synchronize()
        assert np.array_equal(s.getCurrentState(), O.run(g, r, rule, 4)), (n, r)
        s.close()


@pytest.mark.parametrize("radius", [1, 5, 6, 16, 17, 33, 60, 91, 113, 128])
def test_staged_ragged_sides_vs_oracle(radius):
    """Around the side from which ragged rows are staged, with the row's end early, late and
    in the middle of a word and of a tile."""
    import cat_cpu_b200 as C
    rng = np.random.default_rng(50 + radius)
    N = (2 * radius + 1) ** 2
    rule = (int(0.45 * N), N, int(0.45 * N), N)  # above the mean count: domains of both kinds
    for n in (1919, 1921, 1950, 2047, 2049, 2079, 2191):
        g = (rng.random((n, n)) < 0.45).astype(np.uint8)
        with C.CUDASolver(n, radius, rule, variant=C.VARIANT_TENSOR) as s:
            s.setState(g)
            for steps in (2, 1):  # many generations per launch, and one
                s.doSteps(steps)
                s.synchronize()
                g = O.run(g, radius, rule, steps)
                assert np.array_equal(s.getCurrentState(), g), (n, radius, steps)
