"""Solvers of several kinds on streams of their own, launched from several threads
without waiting for one another: the launches whose CTAs wait for one another (small
packed and tensor grids, batches with groups) share the GPU with each other and with
plain ones.  Bit-exact against the oracle, and no bounded wait runs out."""
import threading

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_streams_and_threads():
    import torch
    import cat_cpu_b200 as C
    rounds, steps = 8, 5
    cfg = [(C.VARIANT_PACKED, 1300, 5), (C.VARIANT_TENSOR, 900, 6), (C.VARIANT_PACKED, 700, 3), (C.VARIANT_AUTO, 64, 1),
           (C.VARIANT_PLAIN, 600, 4), (C.VARIANT_TENSOR, 500, 20), (C.VARIANT_PACKED, 1100, 12)]
    rng = np.random.default_rng(4)
    grids, solvers, streams = [], [], []
    for variant, n, r in cfg:
        grids.append((rng.random((n, n)) < 0.45).astype(np.uint8))
        streams.append(torch.cuda.Stream())
        solvers.append(C.CUDASolver(n, r, O.scaled_rule(r), variant=variant))
        solvers[-1].set_stream(streams[-1].cuda_stream)
        solvers[-1].setState(grids[-1])
    sides = [(300, 2), (1000, 5), (64, 1), (700, 8)]
    batch = C.Batch([(n, r, O.scaled_rule(r)) for n, r in sides])
    streams.append(torch.cuda.Stream())
    batch.set_stream(streams[-1].cuda_stream)
    flat = [(rng.random((n, n)) < 0.45).astype(np.uint8) for n, _ in sides]
    batch.upload_all(np.concatenate([g.ravel() for g in flat]))
    errors = []

    def drive(step, finish):
        try:
            for _ in range(rounds):
                step(steps)
            finish()
        except Exception as e:  # an exception in a thread must fail the test
            errors.append(e)

    threads = [threading.Thread(target=drive, args=(s.doSteps, s.synchronize)) for s in solvers]
    threads.append(threading.Thread(target=drive, args=(batch.step, batch.synchronize)))
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (variant, n, r), g, s in zip(cfg, grids, solvers):
        assert np.array_equal(s.getCurrentState(), O.run(g, r, O.scaled_rule(r), rounds * steps)), (variant, n, r)
        s.close()
    got = batch.download_all()
    for k, ((n, r), g) in enumerate(zip(sides, flat)):
        part = got[batch.offsets[k]:batch.offsets[k + 1]].reshape(n, n)
        assert np.array_equal(part, O.run(g, r, O.scaled_rule(r), rounds * steps)), (n, r)
    batch.close()
