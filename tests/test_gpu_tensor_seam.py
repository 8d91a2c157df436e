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
            s.doSteps(2)
            s.synchronize()
            assert np.array_equal(s.getCurrentState(), O.run(g, radius, rule, 2)), (n, radius)
