"""A bounded wait that runs out, in the launches whose CTAs wait for one another (small
packed and tensor grids, batches with groups): whichever call next waits for results
returns LTL_ETIMEOUT, once, and an upload makes the solver whole again, asked or not.
The waits run out because the barrier expects a CTA (the tensor step: a completion
signal) that never comes; the kernels give up after a few ms and return."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# bands in several CTAs, tiles, tensor: gathered, staged with and without a seam
SOLVERS = [("packed", 300, 5), ("packed", 2048, 8), ("tensor", 700, 5), ("tensor", 2001, 5), ("tensor", 704, 5)]
RULE = {5: O.BOSCO_R5}


def rule_of(r):
    return RULE.get(r, O.scaled_rule(r))


def make(kind, n, r):
    import cat_cpu_b200 as C
    s = C.CUDASolver(n, r, rule_of(r), variant=C.VARIANT_PACKED if kind == "packed" else C.VARIANT_TENSOR)
    if kind == "tensor":
        s.set_param("wait_limit_ns", 5_000_000)
    return s


def inject(s, kind, on):
    if kind == "packed":
        s.set_param("inject_missing_arrival", 5_000_000 if on else 0)
    else:
        s.set_param("inject_missing_commit", 1 if on else 0)


def times_out(call):
    import cat_cpu_b200 as C
    with pytest.raises(C.LtlError) as e:
        call()
    assert e.value.code == C.ltl.ETIMEOUT


@pytest.mark.parametrize("kind,n,r", SOLVERS)
def test_every_call_that_waits_reports(kind, n, r):
    import torch
    g = (np.random.default_rng(n).random((n, n)) < 0.45).astype(np.uint8)
    want = O.run(g, r, rule_of(r), 4)
    other = torch.zeros((n, n), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with make(kind, n, r) as s:
        calls = [s.synchronize, s.getCurrentState, s.getCurrentStatePacked, s.population,
                 lambda: s.compare_device(other.data_ptr(), n)]
        for call in calls:
            inject(s, kind, True)
            s.setState(g)
            s.doSteps(4)
            times_out(call)
            s.synchronize()  # reported once
            inject(s, kind, False)
            s.setState(g)
            s.doSteps(4)
            call()
            assert np.array_equal(s.getCurrentState(), want)


@pytest.mark.parametrize("kind,n,r", SOLVERS)
def test_an_upload_heals_what_nobody_asked_for(kind, n, r):
    """The next grid is right, and the lost one is still reported."""
    import torch
    import cat_cpu_b200 as C
    g = (np.random.default_rng(n + 1).random((n, n)) < 0.45).astype(np.uint8)
    want = O.run(g, r, rule_of(r), 6)
    dev, out = torch.from_numpy(g).cuda(), torch.zeros((n, n), dtype=torch.uint8, device="cuda")
    words = C.pack_grid(g)
    torch.cuda.synchronize()
    with make(kind, n, r) as s:
        for put in (lambda: s.setState(g), lambda: s.upload_device(dev.data_ptr(), n), lambda: s.setStatePacked(words)):
            inject(s, kind, True)
            s.setState(g)
            s.doSteps(20)  # (few enough generations would need no barrier)
            inject(s, kind, False)
            put()
            s.doSteps(6)
            s.download_device(out.data_ptr(), n)
            times_out(s.synchronize)
            assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("kind,n,r", SOLVERS)
def test_replays_of_a_captured_step_report(kind, n, r):
    import torch
    g = (np.random.default_rng(n + 2).random((n, n)) < 0.45).astype(np.uint8)
    stream = torch.cuda.Stream()
    with make(kind, n, r) as s:
        s.set_stream(stream.cuda_stream)
        s.setState(g)
        inject(s, kind, True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            s.doSteps(4)
        s.synchronize()  # nothing has run
        for _ in range(2):
            s.setState(g)
            with torch.cuda.stream(stream):
                graph.replay()
            times_out(s.getCurrentState)
        del graph


def test_batch_groups():
    import cat_cpu_b200 as C
    sides = [(1000, 5), (64, 1), (700, 8)]
    rng = np.random.default_rng(9)
    grids = [(rng.random((n, n)) < 0.45).astype(np.uint8) for n, _ in sides]
    want = [O.run(g, r, rule_of(r), 4) for g, (_, r) in zip(grids, sides)]
    flat = np.concatenate([g.ravel() for g in grids])
    for flags in (0, 2):  # through the batch's own graph, and launched directly
        b = C.Batch([(n, r, rule_of(r)) for n, r in sides], flags=flags)
        for call in (b.synchronize, b.download_all, lambda: b.download(0)):
            b.set_param("inject_missing_arrival", 5_000_000)
            b.upload_all(flat)
            b.step(4)
            times_out(call)
            b.synchronize()
            # unasked: another upload comes first
            b.step(4)
            b.set_param("inject_missing_arrival", 0)
            for k, g in enumerate(grids):
                b.upload(k, g)
            b.step(4)
            times_out(b.synchronize)
            got = b.download_all()
            for k, w in enumerate(want):
                assert np.array_equal(got[b.offsets[k]:b.offsets[k + 1]].reshape(w.shape), w), sides[k]
        b.close()


def test_arguments():
    import cat_cpu_b200 as C
    with C.CUDASolver(300, 5, O.BOSCO_R5, variant=C.VARIANT_PACKED) as s:
        for bad in (1, 999_999, 10**10 + 1, -1):
            with pytest.raises(C.LtlError):
                s.set_param("inject_missing_arrival", bad)
    for variant in (C.VARIANT_AUTO, C.VARIANT_PLAIN, C.VARIANT_TENSOR):
        with C.CUDASolver(300, 5, O.BOSCO_R5, variant=variant) as s, pytest.raises(C.LtlError):
            s.set_param("inject_missing_arrival", 10**7)


def test_replays_of_a_captured_batch_report():
    import torch
    import cat_cpu_b200 as C
    n, r = 1000, 5
    flat = (np.random.default_rng(3).random(n * n) < 0.45).astype(np.uint8)
    stream = torch.cuda.Stream()
    b = C.Batch([(n, r, rule_of(r))], flags=2)  # launched directly, so that it can be captured
    b.set_param("inject_missing_arrival", 5_000_000)
    b.set_stream(stream.cuda_stream)
    b.upload_all(flat)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        b.step(4)
    b.synchronize()  # nothing has run
    for _ in range(2):
        b.upload_all(flat)
        with torch.cuda.stream(stream):
            graph.replay()
        times_out(b.download_all)
    del graph
    b.close()
