"""The work a user of this framework has it do, as cases that can be timed and compared.

Three kinds of pass, each through the package's public calls:

  solve   one grid: put the start grid in, advance `steps` generations, take the
          grid out.  `io` is where the grid lives: "device" (a torch tensor,
          upload_device / download_device), "host" (uint8 numpy, setState /
          getCurrentState, the reference's own call sequence) or "packed"
          (uint64 numpy in the PACK coding).  `ask` is what a program asks beside
          the grid: "population" (a live count every `every` generations),
          "compare" (the cell-for-cell check against an expected grid, as
          --doVerify does) or "" (nothing).
  batch   many independent tori of uneven side, radius and rule: upload_all,
          step, download_all on host buffers (the batch API has no other).
  codec   a device grid to PACK words and back (checkpoints, transfers).

Rules: Bosco at R = 5, else the interval rule scaled to the neighbourhood, as in
the package's workloads.  Cells are Bernoulli(density) from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import cat_cpu_b200 as C
from cat_cpu_b200 import workloads

VARIANTS = {"auto": C.VARIANT_AUTO, "plain": C.VARIANT_PLAIN, "tensor": C.VARIANT_TENSOR, "packed": C.VARIANT_PACKED}
_stream = None


def _work_stream():
    """The one side stream a program gives all its solvers."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _solve(name, variant, n, radius, steps, density=0.5, io="device", ask="", every=0):
    c = {"kind": "solve", "variant": variant, "n": n, "radius": radius, "steps": steps, "density": density,
         "io": io, "ask": ask, "every": every}
    return dict(c, name=name) if name else c


def _batch(name, count, nmin, nmax, rmax, steps, seed):
    c = {"kind": "batch", "count": count, "nmin": nmin, "nmax": nmax, "rmax": rmax, "steps": steps, "seed": seed}
    return dict(c, name=name) if name else c


def _codec(name, rows, cols):
    c = {"kind": "codec", "rows": rows, "cols": cols}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: an interactive 64 x 64 torus (the smallest batched side) advanced a few generations
        _solve("tiny_auto_64_r1", "auto", 64, 1, 8),
        # the 1024^2, 100-generation workload, from and to host memory with the default solver, as the reference runs it
        _solve("auto_1024_r5_host", "auto", 1024, 5, 100, io="host"),
        # the same size on the bit-packed solver, device-resident (simulation inside a torch program)
        _solve("packed_1024_r5", "packed", 1024, 5, 100),
        # the headline 16384^2 Bosco grid on each solver
        _solve("plain_16384_r5", "plain", 16384, 5, 100),
        _solve("packed_16384_r5", "packed", 16384, 5, 100),
        _solve("tensor_16384_r5", "tensor", 16384, 5, 100),
        # large radius on the plain solver, a side that no tile divides, checked against an expected grid
        _solve("plain_6001_r64_verify", "plain", 6001, 64, 20, density=0.45, ask="compare"),
        # odd side on the bit-packed solver, PACK-coded host transfers, live count while it runs
        _solve("packed_3001_r8_monitor", "packed", 3001, 8, 64, io="packed", ask="population", every=8),
        # the tensor solver at a middle size and a radius where it is the fastest counted form
        _solve("tensor_4096_r16", "tensor", 4096, 16, 32),
        # a small ensemble and a large one (sides log-uniform in [64, 2048], R in 1..8, 256 generations)
        _batch("batch_64", 64, 64, 2048, 8, 256, 11),
        _batch("batch_1024", 1024, 64, 2048, 8, 256, 4),
        # checkpoint coding of the headline grid
        _codec("codec_16384", 16384, 16384),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A side of the range: two in five a multiple of 64, as configured sizes are, else as drawn."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 0.4:
        n = max(64, n // 64 * 64)
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.random()
    if kind < 0.12:
        rows, cols = _side(rng, 64, 16384), _side(rng, 64, 16384)
        return _codec(None, rows, cols)
    if kind < 0.27:
        count = _log_int(rng, 8, 512)
        nmax = _log_int(rng, 256, 2048)
        return _batch(None, count, 64, nmax, rng.randint(1, 8), _log_int(rng, 16, 256), rng.randint(0, 10**6))
    variant = rng.choice(["auto", "plain", "plain", "packed", "packed", "packed", "tensor", "tensor"])
    if variant in ("auto", "plain"):
        radius = rng.randint(1, 5) if rng.random() < 0.6 else _log_int(rng, 6, 128)
    elif variant == "packed":
        radius = rng.randint(1, 16)
    else:
        radius = _log_int(rng, 1, 64)
    n = _side(rng, max(64, 4 * radius), 16384)
    steps = _log_int(rng, 1, 100)
    # no more cell updates than the headline case, and fewer where a cell costs more
    cost = 1 + radius // 6
    steps = max(1, min(steps, int(100 * 16384**2 / (cost * n * n))))
    io = rng.choice(["device", "device", "device", "host", "packed"])
    ask = rng.choice(["", "", "", "population", "compare"])
    density = 0.5 if radius <= 8 else 0.45
    return _solve(None, variant, n, radius, steps, density, io, ask, max(1, steps // 8) if ask == "population" else 0)


def _rule(radius):
    return workloads.BOSCO_R5 if radius == 5 else workloads.scaled_rule(radius)


def _cells(rows, cols, density, seed):
    """A Bernoulli grid on the GPU, made from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    out = torch.empty((rows, cols), dtype=torch.uint8, device="cuda")
    for r0 in range(0, rows, 4096):
        r1 = min(rows, r0 + 4096)
        out[r0:r1] = torch.rand((r1 - r0, cols), generator=gen, device="cuda") < density
    return out


def _batch_grids(case):
    """[(n, R, rule)] and the densities of a batch: its plan, drawn from the case's own seed."""
    rng = workloads.MT19937_64(case["seed"])
    grids, dens = [], []
    for _ in range(case["count"]):
        u = rng() / 2.0**64
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** u))
        r = 1 + rng() % case["rmax"]
        grids.append((max(case["nmin"], min(case["nmax"], n)), r, workloads.scaled_rule(r)))
        dens.append(0.2 + 0.4 * (rng() / 2.0**64))
    return grids, dens


def _batch_cells(grids, dens, seed):
    sizes = torch.tensor([g[0] * g[0] for g in grids])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    threshold = torch.repeat_interleave(torch.tensor(dens, dtype=torch.float32), sizes).cuda()
    return (torch.rand(threshold.shape, generator=gen, device="cuda") < threshold).to(torch.uint8)


def prepare(case, seed):
    if case["kind"] == "codec":
        rows, cols = case["rows"], case["cols"]
        return {"case": case, "cells": _cells(rows, cols, 0.5, seed),
                "words": torch.zeros((rows, (cols + 63) // 64), dtype=torch.int64, device="cuda"),
                "back": torch.zeros((rows, cols), dtype=torch.uint8, device="cuda")}
    stream = _work_stream()
    if case["kind"] == "batch":
        grids, dens = _batch_grids(case)
        batch = C.Batch(grids)
        batch.set_stream(stream.cuda_stream)
        # pinned host buffers, as a program that moves ensembles keeps them
        cells = torch.empty(int(batch.offsets[-1]), dtype=torch.uint8, pin_memory=True)
        cells.copy_(_batch_cells(grids, dens, seed))
        out = torch.empty_like(cells, pin_memory=True)
        torch.cuda.synchronize()
        return {"case": case, "batch": batch, "cells": cells.numpy(), "out": out.numpy(), "keep": (cells, out)}
    n, radius = case["n"], case["radius"]
    solver = C.CUDASolver(n, radius, _rule(radius), variant=VARIANTS[case["variant"]])
    solver.set_stream(stream.cuda_stream)
    state = {"case": case, "solver": solver, "grid": _cells(n, n, case["density"], seed)}
    if case["ask"] == "compare":
        # the expected grid: another run's, here an independent one of the same density
        state["expected"] = _cells(n, n, case["density"], seed + 1000003)
    if case["io"] == "device":
        state["out"] = torch.zeros((n, n), dtype=torch.uint8, device="cuda")
    else:
        host = state["grid"].cpu().numpy()
        state["host"] = host if case["io"] == "host" else C.pack_grid(host)
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "codec":
        return _run_codec(state)
    if case["kind"] == "batch":
        state["batch"].upload_all(state["cells"])
        state["batch"].step(case["steps"])
        return state["batch"].download_all(state["out"])
    s, n, left = state["solver"], case["n"], case["steps"]
    if case["io"] == "device":
        s.upload_device(state["grid"].data_ptr(), n)
    elif case["io"] == "host":
        s.setState(state["host"])
    else:
        s.setStatePacked(state["host"])
    out = {}
    if case["ask"] == "population":
        live = []
        while left > 0:
            k = min(case["every"], left)
            s.doSteps(k)
            live.append(s.population())
            left -= k
        out["live"] = np.array(live, dtype=np.int64)
    else:
        s.doSteps(left)
    if case["ask"] == "compare":
        out["mismatches"], out["first"] = s.compare_device(state["expected"].data_ptr(), n)
    if case["io"] == "device":
        s.download_device(state["out"].data_ptr(), n)
        out["grid"] = state["out"]
    elif case["io"] == "host":
        out["grid"] = s.getCurrentState()
    else:
        out["grid"] = s.getCurrentStatePacked().view(np.int64)
    return out


def _run_codec(state):
    lib, stream = C.lib(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    cells, words, back = state["cells"], state["words"], state["back"]
    rows, cols = cells.shape
    pitch = words.shape[1] * 8
    C.ltl.check(lib.ltl_pack_device(ctypes.c_void_p(cells.data_ptr()), cols, rows, cols,
                                    ctypes.c_void_p(words.data_ptr()), pitch, stream))
    C.ltl.check(lib.ltl_unpack_device(ctypes.c_void_p(words.data_ptr()), pitch, rows, cols,
                                      ctypes.c_void_p(back.data_ptr()), cols, stream))
    return {"words": words, "cells": back}


def _cell_updates(case):
    if case["kind"] == "solve":
        return case["n"] ** 2 * case["steps"]
    return sum(g[0] ** 2 for g in _batch_grids(case)[0]) * case["steps"]


def work(case):
    """Bytes: the grid in and out once in the coding it comes in (generations in between need not
    leave the chip).  Operations: per cell update the four adds of the two sliding sums and the
    four comparisons of the rule."""
    if case["kind"] == "codec":
        cells = case["rows"] * case["cols"]
        words = 8 * case["rows"] * ((case["cols"] + 63) // 64)
        return {"bytes": 2 * cells + 2 * words, "flops": 0}
    cells = _cell_updates(case) // case["steps"]
    per_cell = 0.25 if case.get("io") == "packed" else 2.0
    more = cells if case.get("ask") == "compare" else 0
    return {"bytes": per_cell * cells + more, "flops": 8.0 * _cell_updates(case)}


def _step64(grid, radius, rule):
    """One generation in plain torch, 64-bit sums (box count by padded cumulative sums)."""
    smin, smax, bmin, bmax = rule
    count = grid
    for dim in (0, 1):
        first, last = count.narrow(dim, 0, radius), count.narrow(dim, count.shape[dim] - radius, radius)
        wide = torch.cat([last, count, first], dim)
        total = torch.cumsum(wide, dim, dtype=torch.int64)
        total = torch.cat([torch.zeros_like(total.narrow(dim, 0, 1)), total], dim)
        size, span = grid.shape[dim], 2 * radius + 1
        count = total.narrow(dim, span, size) - total.narrow(dim, 0, size)
    count = count - grid
    lives = (count >= smin) & (count <= smax)
    born = (count >= bmin) & (count <= bmax)
    return torch.where(grid > 0, lives, born).to(torch.int64)


def _pack64(grid):
    return C.pack_grid(grid.to(torch.uint8).cpu().numpy()).view(np.int64)


def exact(case, seed):
    if case["kind"] == "codec":
        cells = _cells(case["rows"], case["cols"], 0.5, seed)
        return {"words": _pack64(cells), "cells": cells}
    if _cell_updates(case) > 3 * 10**10:
        return None
    if case["kind"] == "batch":
        grids, dens = _batch_grids(case)
        if case["count"] * case["steps"] > 20000:
            return None
        flat, out, at = _batch_cells(grids, dens, seed), [], 0
        for n, radius, rule in grids:
            g = flat[at:at + n * n].view(n, n).to(torch.int64)
            at += n * n
            for _ in range(case["steps"]):
                g = _step64(g, radius, rule)
            out.append(g.to(torch.uint8).reshape(-1))
        return torch.cat(out).cpu().numpy()
    n, radius = case["n"], case["radius"]
    g = _cells(n, n, case["density"], seed).to(torch.int64)
    out, live = {}, []
    for k in range(case["steps"]):
        g = _step64(g, radius, _rule(radius))
        if case["ask"] == "population" and ((k + 1) % case["every"] == 0 or k + 1 == case["steps"]):
            live.append(int(g.sum()))
    if case["ask"] == "population":
        out["live"] = np.array(live, dtype=np.int64)
    if case["ask"] == "compare":
        differ = (g != _cells(n, n, case["density"], seed + 1000003)).reshape(-1)
        out["mismatches"] = int(differ.sum())
        out["first"] = int(torch.argmax(differ.to(torch.uint8))) if out["mismatches"] else -1
    out["grid"] = _pack64(g) if case["io"] == "packed" else g.to(torch.uint8)
    return out
