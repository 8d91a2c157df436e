"""A solver's first launches while the device's default stream is still busy: what they
expect to be zero was zeroed in their own stream, which does not wait for that one.
Bit-exact against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def busy_default_stream():
    """Leaves freed device memory full of ones, then about 0.3 s of work."""
    import torch
    x = torch.full((256 << 20,), -1, dtype=torch.int8, device="cuda")
    torch.cuda.synchronize()
    del x
    torch.cuda.empty_cache()
    torch.cuda._sleep(500_000_000)


@pytest.mark.parametrize("variant", [1, 2])
def test_first_steps_of_a_solver(variant):
    import torch
    import cat_cpu_b200 as C
    n, r = 700, 5
    g = (np.random.default_rng(3).random((n, n)) < 0.45).astype(np.uint8)
    want = O.run(g, r, O.BOSCO_R5, 6)
    busy_default_stream()
    with C.CUDASolver(n, r, O.BOSCO_R5, variant=variant) as s:
        s.setState(g)
        s.doSteps(6)
        s.synchronize()
        got = s.getCurrentState()
    torch.cuda.synchronize()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("persistent", [1, 0])
def test_first_steps_of_a_batch(persistent):
    import torch
    import cat_cpu_b200 as C
    sides = [(900, 4), (64, 1), (300, 7)]
    rng = np.random.default_rng(5)
    grids = [(rng.random((n, n)) < 0.45).astype(np.uint8) for n, _ in sides]
    want = [O.run(g, r, O.scaled_rule(r), 5) for g, (_, r) in zip(grids, sides)]
    busy_default_stream()
    b = C.Batch([(n, r, O.scaled_rule(r)) for n, r in sides])
    b.set_param("persistent", persistent)
    b.upload_all(np.concatenate([g.ravel() for g in grids]))
    b.step(5)
    got = b.download_all()
    torch.cuda.synchronize()
    for k, w in enumerate(want):
        assert np.array_equal(got[b.offsets[k]:b.offsets[k + 1]].reshape(w.shape), w), sides[k]
    b.close()
