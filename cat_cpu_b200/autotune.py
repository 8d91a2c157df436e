"""Shape autotuner: sweeps the kernels' work-item shapes on the device, against the
shapes that are built in, and writes those that beat them to
cat_cpu_b200/tuning/ltl_tuning.txt, which libltl_b200 reads at ltl_create /
ltl_batch_create.

    python -m cat_cpu_b200.autotune [--quick] [--out DIR]

This is the analogue of the reference project's region-count landscape search
(NREGIONS_H/V over 1..30 x 1..30, scripts/exploreRegionSizesLandscape.py:21-39,
scripts/extractBestRegionSize.py): here the swept shapes are
  plain / packed   band_rows: rows a warp walks down per work item (the vertical
                   window is restarted once per band, so longer bands re-read less
                   but leave fewer items to balance over 148 SMs); 0 is the
                   built-in choice, which follows the grid's sides;
  plain            depth: generations per pass of the temporally blocked kernel
                   (1, 2 or 3), swept jointly with band_rows;
  batch            persistent: one launch per call that runs every generation of
                   every grid (1), or per-generation launches (0), and for the
                   latter stream_band_rows of the streamed per-step kernels and
                   resident_max_bytes: which grids are kept in shared memory for
                   a whole multi-step launch and which are streamed each step.
A line of the table holds for a class of sides, so a shape gets one only if it is
faster than the built-in choice at every side of the class that was timed, and by
more than MARGIN on average.  The full landscape (every candidate's time) is written
next to the table.
"""
import argparse
import concurrent.futures as cf
import os
import time

import numpy as np

PKG = os.path.dirname(os.path.abspath(__file__))
MARGIN = 0.03


def choose(times, builtin):
    """The candidate to write for a class of sides, or None to leave it to the built-in
    choice.  times: {side: {candidate: ms}}, `builtin` among the candidates."""
    gains = {}
    for cand in next(iter(times.values())):
        ratio = [t[cand] / t[builtin] for t in times.values()]
        if cand != builtin and max(ratio) < 1:
            gains[cand] = float(np.exp(np.mean(np.log(ratio))))
    best = min(gains, key=gains.get, default=None)
    return best if best is not None and gains[best] < 1 - MARGIN else None


def _time_steps(torch, solver, stream, steps, reps=3):
    best = None
    for _ in range(reps):
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record(stream)
        solver.doSteps(steps)
        b.record(stream)
        stream.synchronize()
        ms = a.elapsed_time(b) / steps
        best = ms if best is None else min(best, ms)
    return best


def size_class(n):
    """Grid-side class a tuned value applies to: [1, 8191], [8192, 24575], [24576, 2^30]."""
    if n < 8192:
        return 1, 8191
    if n < 24576:
        return 8192, 24575
    return 24576, 1 << 30


def tune_single(torch, C, variant, n, radius, rule, candidates, steps, depths=(1,)):
    """{(depth, band_rows): ms per step} and the built-in pair; `steps` should be a multiple
    of every depth."""
    vcode = {"plain": C.VARIANT_PLAIN, "packed": C.VARIANT_PACKED}[variant]
    g = C.generate_state(n, 12345, 0.5, 1)
    stream = torch.cuda.Stream()
    s = C.CUDASolver(n, radius, rule, variant=vcode)
    s.set_stream(stream.cuda_stream)
    builtin = (s.info.temporal_depth, 0)
    times = {}
    try:
        for d in depths:
            if variant == "plain":
                s.set_param("depth", d)
            for br in candidates:
                s.set_param("band_rows", br)
                s.setState(g)
                s.doSteps(12)
                times[(d, br)] = _time_steps(torch, s, stream, steps)
    finally:
        s.close()
    return times, builtin


def tune_batch(torch, C, band_candidates, resident_candidates, steps):
    from cat_cpu_b200.workloads import batch_config
    cfg = batch_config()
    with cf.ThreadPoolExecutor(os.cpu_count() or 8) as ex:
        grids = list(ex.map(lambda c: C.generate_state(c[0], c[4], c[3], 1), cfg))
    flat = np.concatenate([g.ravel() for g in grids])
    stream = torch.cuda.Stream()
    b = C.Batch([(n, r, rule) for (n, r, rule, d, s) in cfg])
    rows = []
    try:
        b.set_stream(stream.cuda_stream)
        # (persistent, stream_band_rows, resident_max_bytes); the last two only
        # matter for per-generation launches
        cands = [(1, band_candidates[0], resident_candidates[0])] + \
            [(0, br, rm) for rm in resident_candidates for br in band_candidates]
        for pers, br, rm in cands:
            b.set_param("persistent", pers)
            b.set_param("resident_max_bytes", rm)
            b.set_param("stream_band_rows", br)
            b.upload_all(flat)
            b.step(steps)          # builds and warms the graph
            b.synchronize()
            a = torch.cuda.Event(enable_timing=True)
            e = torch.cuda.Event(enable_timing=True)
            a.record(stream)
            b.step(steps)
            e.record(stream)
            stream.synchronize()
            rows.append(((pers, br, rm), a.elapsed_time(e)))
    finally:
        b.close()
    return dict(rows), cands[0]


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--quick", action="store_true", help="fewer candidates")
    ap.add_argument("--out", default=os.path.join(PKG, "tuning"))
    args = ap.parse_args()
    os.environ["LTL_TUNING_FILE"] = os.devnull  # the built-in choices, not an earlier table's
    import torch
    import cat_cpu_b200 as C
    from cat_cpu_b200.workloads import scaled_rule, BOSCO_R5

    os.makedirs(args.out, exist_ok=True)
    dev = torch.cuda.get_device_name(0)
    table = [f"# shapes that beat the built-in ones on {dev}: cat_cpu_b200/autotune.py, {time.strftime('%Y-%m-%d %H:%M:%S')}"]
    land = [f"# landscape ({dev}): candidate -> ms per step (single grids) or per 256-step batch run"]
    bands = [0, 16, 64, 256] if args.quick else [0, 16, 32, 48, 64, 96, 128, 192, 256, 384, 512]  # 0: built-in
    sides = [(1024, 4096), (8192, 16384), (32768,)]  # of each class
    jobs = [("plain", 5), ("packed", 5)] + ([] if args.quick else [("plain", 1)] + [("packed", r) for r in (1, 2, 8, 16, 32)])
    for variant, r in jobs:
        rule = BOSCO_R5 if r == 5 else scaled_rule(r)
        depths = [d for d in (1, 2, 3) if d == 1 or (r <= 5 and d * r <= 16)] if variant == "plain" else [1]
        for ns in sides:
            times = {}
            for n in ns:
                times[n], builtin = tune_single(torch, C, variant, n, r, rule, bands, 24, depths)
                land.append(f"{variant} n={n} R={r} (depth, band_rows): " +
                            ", ".join(f"{c}:{t:.4f}" for c, t in times[n].items()) + f"  built-in {builtin}")
                print(land[-1], flush=True)
            best = choose(times, builtin)
            if best is not None:
                lo, hi = size_class(ns[0])
                extra = f" depth={best[0]}" if variant == "plain" else ""
                table.append(f"variant={variant} radius={r} nmin={lo} nmax={hi} band_rows={best[1]}{extra}")
                print("->", table[-1], flush=True)
    band_c = [32, 64, 128] if args.quick else [32, 48, 64, 96, 128]
    res_c = [0, 225280] if args.quick else [0, 65536, 131072, 225280]
    times, builtin = tune_batch(torch, C, band_c, res_c, 256)
    land.append("batch (persistent, stream_band_rows, resident_max_bytes): " +
                ", ".join(f"{c}:{t:.2f}" for c, t in times.items()))
    print(land[-1], flush=True)
    # of the per-generation shapes the best one is written in any case: callers choose that mode
    pers = choose({0: times}, builtin) is None
    _, br, rm = min((c for c in times if c[0] == 0), key=times.get)
    table.append(f"variant=batch radius=* persistent={int(pers)} stream_band_rows={br} resident_max_bytes={rm}")
    with open(os.path.join(args.out, "ltl_tuning.txt"), "w") as f:
        f.write("\n".join(table) + "\n")
    with open(os.path.join(args.out, "landscape.txt"), "w") as f:
        f.write("\n".join(land) + "\n")
    print("wrote", os.path.join(args.out, "ltl_tuning.txt"))


if __name__ == "__main__":
    main()
