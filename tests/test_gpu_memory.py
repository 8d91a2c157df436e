"""Transfers, and the steps between them, with the device's memory taken: a solver that
was made needs no more of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fill_memory():
    """Takes the device's free memory, down to pieces of about 20 MB."""
    import torch
    held = []
    for size in (1 << 33, 1 << 30, 1 << 27, 1 << 25, 21 << 20):
        while True:
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    return held


@pytest.mark.parametrize("variant,n,packed_too", [(0, 16001, False), (2, 16001, True), (-1, 16001, True), (1, 16001, True),
                                                  (-1, 16384, True)])
def test_transfers_when_memory_is_taken(variant, n, packed_too):
    """16001^2 cells are 256 MB, in the PACK coding 32 MB."""
    import torch
    import cat_cpu_b200 as C
    rule = (2, 3, 3, 3)

    def go(s, g):
        s.setState(g * 85)  # any byte but 0 is a live cell
        a = s.getCurrentState()
        s.doSteps(3)
        s.synchronize()
        b = s.getCurrentState()
        p = None
        if packed_too:
            s.setStatePacked(C.pack_grid(g))
            p = s.getCurrentStatePacked()
        return a, b, p

    rng = np.random.default_rng(n)
    small = (rng.random((n % 16 + 2000, n % 16 + 2000)) < 0.4).astype(np.uint8)
    g = np.tile(small, (9, 9))[:n, :n].copy()
    with C.CUDASolver(n, 1, rule, variant=variant) as s, C.CUDASolver(n, 1, rule, variant=2) as other:
        want = go(s, g)  # loads the kernels
        assert np.array_equal(want[0], g)
        other.setState(g)
        other.doSteps(3)
        assert np.array_equal(other.getCurrentState(), want[1])
    with C.CUDASolver(n, 1, rule, variant=variant) as s:
        held = fill_memory()
        try:
            got = go(s, g)
        finally:
            del held
            torch.cuda.empty_cache()
        assert np.array_equal(got[0], g) and np.array_equal(got[1], want[1])
        assert not packed_too or np.array_equal(got[2], C.pack_grid(g))


@pytest.mark.parametrize("n,radius", [(64, 1), (1000, 5), (4097, 28), (16384, 5)])
def test_default_solver_holds_no_more_than_the_plain_one(n, radius):
    import cat_cpu_b200 as C
    rule = (2, 3, 3, 3)
    with C.CUDASolver(n, radius, rule) as s, C.CUDASolver(n, radius, rule, variant=C.VARIANT_PLAIN) as p:
        assert s.info.device_bytes <= p.info.device_bytes


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_a_solver_that_does_not_fit_leaves_others_alone(variant):
    import cat_cpu_b200 as C
    from oracle import oracle as O
    g = (np.random.default_rng(2).random((500, 500)) < 0.45).astype(np.uint8)
    rule = O.scaled_rule(3)
    with C.CUDASolver(500, 3, rule, variant=variant) as s:
        s.setState(g)
        for make in (lambda: C.CUDASolver(450000, 3, rule, variant=0), lambda: C.Batch([(400000, 3, rule)])):
            with pytest.raises(C.LtlError) as e:
                make()
            assert e.value.code == C.ltl.ENOMEM
            s.doSteps(1)
            g = O.run(g, 3, rule, 1)
            assert np.array_equal(s.getCurrentState(), g)
