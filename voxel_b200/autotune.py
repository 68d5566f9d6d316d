"""Autotuner for the library's launch-shape knobs (vx_tuning_*).

    python -m voxel_b200.autotune [--quick] [--out PATH]

Times every allowed value of each knob on a representative workload on the
current GPU and writes the fastest settings to voxel_b200/tuning/<device>.json,
which the library applies when it is first loaded on that kind of device:

  * sort.items_u32 / sort.items_u64 / sort.early_counts / sort.rank_ballots /
    sort.radix_bits: radix-sort partition tile size (items per thread, hence
    blocks per SM), whether a tile publishes its digit counts before or after
    ranking, whether keys are ranked with per-bit ballots or a shared-memory
    atomic OR per digit, and the digit width (6, 7 or 8 bits: 6, 5 or 4
    passes over 32-bit keys); timed on 2^26
    u32 and 2^25 60-bit u64 key/value pairs;
  * scan.tile_kb: the prefix sum's tile (32, 16 or 8 KB, with 6, 12 or 24
    resident blocks per SM); timed on 2^28 u32;
  * edit.big_item / edit.blocks_per_sm / edit.leafparent_blocks /
    edit.leafparent_prefetch: the primitive-list length above which a work
    item is expanded by a block or a cluster of blocks, the grid of the edit
    pipelines' item kernels, and the resident blocks and next-node prefetch
    of the DAG leaf-parent kernel; timed on the batched Hash DAG edit of the
    benchmark (16384^3 cave terrain at scale 64, 16,384 spheres of radius
    log-uniform in [1, 256], 60 % add);
  * edit.leafparent_lanes: the threads per leaf-parent item in small edits
    (one cooperative launch); timed on do and undo of 1, 8, 32 and 128
    spheres and boxes of radius up to 128 on a 2048^3 Hash DAG;
  * edit.small_max_voxels: the longest voxel list that runs as one
    cooperative launch; timed on lists of 2,000 to 54,000 voxels, placed in
    and removed from a Hash DAG and an SVO: brush strokes (the voxels of a
    sphere, which gain from it) and voxels all over the world (a leaf each,
    which lose);
  * serve.blocks_per_sm: the grid of the serving loop's edit graphs.

A setting replaces the default only when it is more than 4 % faster.

Every setting's output is compared with the default setting's (the sorted
arrays bit for bit, the edited DAG by 2^20 point queries) before its time
counts, so a setting that computed something else is reported, not chosen.
"""
from __future__ import annotations

import argparse
import itertools
import json
import time

import numpy as np
import torch

from . import lib
from . import api as vx
from . import tuning_file


def _time(fn, reps: int, before=None) -> float:
    """Median device time of fn() in ms (before() runs untimed each rep)."""
    ts = []
    for i in range(reps + 1):
        if before is not None:
            before()
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        if i:  # the first run warms up
            ts.append(a.elapsed_time(b))
    return float(np.median(ts))


def _pick(times: dict, default):
    """The fastest setting, or the default where nothing is faster by more
    than the runs of one setting differ."""
    times = {k: t for k, t in times.items() if t is not None}
    best = min(times, key=times.get)
    return default if default in times and times[default] <= 1.04 * times[best] else best


def tune_sort(n32: int, n64: int, reps: int, log) -> tuple[dict, dict]:
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    cases = {
        "u32": (torch.randint(-(1 << 31), (1 << 31) - 1, (n32,), dtype=torch.int32,
                              device="cuda", generator=g), 32, "sort.items_u32"),
        "u64": (torch.randint(0, 1 << 60, (n64,), dtype=torch.int64, device="cuda",
                              generator=g), 60, "sort.items_u64"),
    }
    times: dict = {}
    for label, (keys0, bits, knob) in cases.items():
        n = keys0.numel()
        vals0 = torch.arange(n, dtype=torch.int32, device="cuda")
        ws = torch.empty(lib().vx_sort_workspace_size(n, keys0.element_size()),
                         dtype=torch.uint8, device="cuda")
        k, v = keys0.clone(), vals0.clone()

        def restore():
            k.copy_(keys0)
            v.copy_(vals0)

        vx.reset_tuning()
        restore()
        vx.sort_pairs(k, v, bits, ws)
        ref_k, ref_v = k.clone(), v.clone()
        for items, early, ballots, radix in itertools.product(
                vx.tuning_options(knob), vx.tuning_options("sort.early_counts"),
                vx.tuning_options("sort.rank_ballots"), vx.tuning_options("sort.radix_bits")):
            vx.set_tuning(knob, items)
            vx.set_tuning("sort.early_counts", early)
            vx.set_tuning("sort.rank_ballots", ballots)
            vx.set_tuning("sort.radix_bits", radix)
            restore()
            vx.sort_pairs(k, v, bits, ws)
            same = bool(torch.equal(k, ref_k) and torch.equal(v, ref_v))
            ms = _time(lambda: vx.sort_pairs(k, v, bits, ws), reps, restore) if same else None
            times[(label, items, early, ballots, radix)] = ms
            log(f"  sort {label} items={items} early={early} ballots={ballots} radix={radix}: "
                + (f"{ms:.3f} ms" if same else "DIFFERENT OUTPUT (not used)"))
    vx.reset_tuning()
    # early / ballots / digit width are shared by both key widths: pick the
    # triple with the least total time (each width at its best items); then
    # items per width.
    best: dict = {}
    score = {}
    for early, ballots, radix in itertools.product(vx.tuning_options("sort.early_counts"),
                                                   vx.tuning_options("sort.rank_ballots"),
                                                   vx.tuning_options("sort.radix_bits")):
        tot = 0.0
        for label, (_, _, knob) in cases.items():
            cand = [times[(label, i, early, ballots, radix)] for i in vx.tuning_options(knob)]
            cand = [c for c in cand if c is not None]
            tot = tot + min(cand) if cand else float("inf")
        score[(early, ballots, radix)] = tot
    now = vx.tuning()
    early, ballots, radix = _pick(score, tuple(now[k] for k in (
        "sort.early_counts", "sort.rank_ballots", "sort.radix_bits")))
    best["sort.early_counts"], best["sort.rank_ballots"] = early, ballots
    best["sort.radix_bits"] = radix
    for label, (_, _, knob) in cases.items():
        opts = {i: times[(label, i, early, ballots, radix)] for i in vx.tuning_options(knob)}
        best[knob] = _pick(opts, now[knob])
    return best, {f"{l} items={i} early={e} ballots={b} radix={r}": t
                  for (l, i, e, b, r), t in times.items()}


def tune_scan(n: int, reps: int, log) -> tuple[dict, dict]:
    """scan.tile_kb: exclusive sum of n u32 (inputs larger than L2), each
    tile shape's output compared with the default shape's."""
    g = torch.Generator(device="cuda")
    g.manual_seed(13)
    data0 = torch.randint(0, 1 << 20, (n,), dtype=torch.int32, device="cuda", generator=g)
    ws = torch.empty(lib().vx_scan_workspace_size(n), dtype=torch.uint8, device="cuda")
    d = data0.clone()
    vx.reset_tuning()
    vx.exclusive_sum(d, ws)
    ref = d.clone()
    times: dict = {}
    for kb in vx.tuning_options("scan.tile_kb"):
        vx.set_tuning("scan.tile_kb", kb)
        d.copy_(data0)
        vx.exclusive_sum(d, ws)
        same = bool(torch.equal(d, ref))
        ms = _time(lambda: vx.exclusive_sum(d, ws), reps, lambda: d.copy_(data0)) if same else None
        times[f"tile_kb={kb}"] = ms
        log(f"  scan u32 tile_kb={kb}: " + (f"{ms:.3f} ms" if same else "DIFFERENT OUTPUT (not used)"))
    vx.reset_tuning()
    valid = {int(k.split("=")[1]): t for k, t in times.items()}
    return {"scan.tile_kb": _pick(valid, vx.tuning()["scan.tile_kb"])}, times


def tune_edit(depth: int, scale: int, count: int, reps: int, log, max_nodes: int,
              arena: int) -> tuple[dict, dict]:
    prims = vx.prims_to_device(vx.config_c4_edits(count, seed=7, world_exp=depth + 2), "cuda")
    pristine = vx.HashDag(depth, max_nodes, arena)
    pristine.build_terrain(7, scale, True)
    if pristine.status() != 0:
        raise RuntimeError("terrain build failed")
    work = vx.HashDag(depth, max_nodes, arena)
    g = torch.Generator(device="cuda")
    g.manual_seed(12)
    pts = torch.randint(0, 4 << depth, (1 << 20, 3), dtype=torch.int32, device="cuda",
                        generator=g)
    vx.reset_tuning()
    work.copy_from(pristine)
    work.apply_primitives(prims)
    if work.status() != 0:
        raise RuntimeError("reference edit failed")
    ref = work.query(pts)
    times: dict = {}

    def measure(big, bps, lpb, pf):
        vx.set_tuning("edit.big_item", big)
        vx.set_tuning("edit.blocks_per_sm", bps)
        vx.set_tuning("edit.leafparent_blocks", lpb)
        vx.set_tuning("edit.leafparent_prefetch", pf)
        work.copy_from(pristine)
        work.apply_primitives(prims)
        ok = work.status() == 0 and bool(torch.equal(work.query(pts), ref))
        ms = _time(lambda: work.apply_primitives(prims), reps,
                   lambda: work.copy_from(pristine)) if ok else None
        if ok and work.status() != 0:
            ms = None
        key = (f"big_item={big} blocks_per_sm={bps} leafparent_blocks={lpb} "
               f"leafparent_prefetch={pf}")
        times[key] = ms
        log(f"  edit {key}: "
            + (f"{ms:.3f} ms" if ms is not None else "FAILED OR DIFFERENT (not used)"))
        return ms

    # Stage 1: long-list threshold and grid.
    now = vx.tuning()
    lpb0, pf0 = now["edit.leafparent_blocks"], now["edit.leafparent_prefetch"]
    stage1 = {(big, bps): measure(big, bps, lpb0, pf0)
              for big, bps in itertools.product(vx.tuning_options("edit.big_item"),
                                                vx.tuning_options("edit.blocks_per_sm"))}
    big, bps = _pick(stage1, (now["edit.big_item"], now["edit.blocks_per_sm"]))
    # Stage 2: resident blocks and next-node prefetch of the leaf-parent
    # kernel at that setting.
    stage2 = {(lpb, pf): measure(big, bps, lpb, pf)
              for lpb, pf in itertools.product(vx.tuning_options("edit.leafparent_blocks"),
                                               vx.tuning_options("edit.leafparent_prefetch"))}
    lpb, pf = _pick(stage2, (lpb0, pf0))
    vx.reset_tuning()
    return {"edit.big_item": big, "edit.blocks_per_sm": bps,
            "edit.leafparent_blocks": lpb, "edit.leafparent_prefetch": pf}, times


def _geomean(ts) -> float:
    return float(np.exp(np.mean(np.log(ts))))


def tune_small(depth: int, scale: int, strokes, reps: int, log, max_nodes: int,
               arena: int) -> tuple[dict, dict]:
    """edit.leafparent_lanes and edit.small_max_voxels: geometric means over
    small edits and over voxel lists; each setting's result is compared by
    point queries with the default's."""
    g = torch.Generator(device="cuda")
    g.manual_seed(14)
    pts = torch.randint(0, 4 << depth, (1 << 18, 3), dtype=torch.int32, device="cuda",
                        generator=g)
    dag = vx.HashDag(depth, max_nodes, arena)
    dag.build_terrain(7, scale, True)
    svo = vx.Svo(depth, 2 * max_nodes, 8 * max_nodes, arena_bytes=arena)
    svo.build_terrain(7, scale, True)
    if dag.status() != 0 or svo.status() != 0:
        raise RuntimeError("terrain build failed")
    times: dict = {}
    now = vx.tuning()

    def sweep(knob, calls, look):
        """calls: {name: fn}; look(): what the calls leave, to compare."""
        ref, means = None, {}
        for v in [now[knob]] + [v for v in vx.tuning_options(knob) if v != now[knob]]:
            vx.set_tuning(knob, v)
            ts = []
            for name, fn in calls.items():
                ts.append(_time(fn, reps))
                times[f"{knob}={v} {name}"] = ts[-1]
            got = look()
            ref = got if ref is None else ref
            means[v] = _geomean(ts) if torch.equal(got, ref) else None
            log(f"  {knob}={v}: "
                + (f"{means[v]:.4f} ms" if means[v] is not None else "DIFFERENT (not used)"))
        vx.reset_tuning()
        return _pick(means, now[knob])

    def edits(n):
        do = vx.generate_primitives(depth + 2, n, 8, sphere_permille=500, add_permille=500,
                                    r_min=1, r_max=128, log_uniform=True)
        undo = do.copy()
        undo["flags"] ^= 1 << 8
        a, b = vx.prims_to_device(do, "cuda"), vx.prims_to_device(undo, "cuda")

        def run():
            dag.apply_primitives(a)
            dag.apply_primitives(b)
        return run

    lanes = sweep("edit.leafparent_lanes", {f"{n} primitives": edits(n) for n in (1, 8, 32, 128)},
                  lambda: dag.query(pts))

    def strokes_and_scatter(world):
        for r in strokes:
            prim = np.zeros(1, vx.PRIM_DTYPE)
            prim["c"][0] = (2 << depth) - 3
            prim["r"][0, 0] = r
            prim["flags"] = vx.make_flags(0, 1)
            vox, _ = vx.rasterize(vx.prims_to_device(prim, "cuda"), depth + 2)
            n = vox.shape[0]
            scattered = torch.randint(0, 4 << depth, (n, 3), dtype=vox.dtype, device="cuda",
                                      generator=g)
            order = torch.randperm(n, device="cuda", generator=g)
            for kind, v in (("stroke", vox[order].contiguous()), ("scattered", scattered)):
                def run(v=v):
                    if world.apply_voxels(v, 1) != 0 or world.apply_voxels(v, 0) != 0:
                        raise RuntimeError("voxel list failed")
                yield f"{type(world).__name__} {kind} {n}", run

    voxels = sweep("edit.small_max_voxels",
                   {**dict(strokes_and_scatter(dag)), **dict(strokes_and_scatter(svo))},
                   lambda: torch.cat([dag.query(pts), svo.query(pts)]))
    return {"edit.leafparent_lanes": lanes, "edit.small_max_voxels": voxels}, times


def tune_serve(depth: int, scale: int, batch: int, reps: int, log, max_nodes: int,
               arena: int) -> tuple[dict, dict]:
    """serve.blocks_per_sm: latency of one small batch (the serving loop's
    typical size) replayed as a graph with a device-side count, on the served
    terrain; the same pipeline the serving loop captures."""
    prims = vx.generate_primitives(depth + 2, batch, 8, sphere_permille=500, add_permille=500,
                                   r_min=1, r_max=128, log_uniform=True)
    buf = vx.prims_to_device(prims, "cuda")
    cnt = torch.tensor([batch], dtype=torch.int32, device="cuda")
    pristine = vx.HashDag(depth, max_nodes, arena)
    pristine.build_terrain(8, scale, True)
    if pristine.status() != 0:
        raise RuntimeError("terrain build failed")
    work = vx.HashDag(depth, max_nodes, arena)
    times: dict = {}
    for bps in vx.tuning_options("serve.blocks_per_sm"):
        vx.set_tuning("edit.blocks_per_sm", bps)  # the serving graphs' grid
        graph = work.graph_primitives(buf, cnt, batch)
        work.copy_from(pristine)
        graph.launch()
        ok = work.status() == 0
        ms = _time(graph.launch, reps, lambda: work.copy_from(pristine)) if ok else None
        graph.close()
        times[f"blocks_per_sm={bps}"] = ms
        log(f"  serve batch of {batch} blocks_per_sm={bps}: "
            + (f"{ms:.3f} ms" if ms is not None else "FAILED (not used)"))
    vx.reset_tuning()
    valid = {int(k.split("=")[1]): t for k, t in times.items()}
    return {"serve.blocks_per_sm": _pick(valid, vx.tuning()["serve.blocks_per_sm"])}, times


def main(argv=None) -> dict:
    ap = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    ap.add_argument("--quick", action="store_true", help="small sizes (a test run)")
    ap.add_argument("--out", default=None, help="output JSON (default: the device's file)")
    ap.add_argument("--quiet", action="store_true")
    args = ap.parse_args(argv)
    log = (lambda m: None) if args.quiet else (lambda m: print(m, flush=True))
    if not torch.cuda.is_available():
        raise SystemExit("autotune needs a CUDA device")
    dev = torch.cuda.get_device_name()
    t0 = time.time()
    if args.quick:
        sort_best, sort_t = tune_sort(1 << 20, 1 << 19, 2, log)
        scan_best, scan_t = tune_scan(1 << 20, 2, log)
        edit_best, edit_t = tune_edit(6, 1, 256, 2, log, 1 << 18, 64 << 20)
        small_best, small_t = tune_small(6, 1, (5, 12), 2, log, 1 << 18, 64 << 20)
        serve_best, serve_t = tune_serve(6, 1, 64, 2, log, 1 << 18, 64 << 20)
    else:
        sort_best, sort_t = tune_sort(1 << 26, 1 << 25, 5, log)
        scan_best, scan_t = tune_scan(1 << 28, 5, log)
        edit_best, edit_t = tune_edit(12, 64, 16384, 5, log, 1 << 27, 16 << 30)
        small_best, small_t = tune_small(9, 8, (8, 12, 16, 20, 23), 15, log, 1 << 22, 2 << 30)
        serve_best, serve_t = tune_serve(11, 32, 400, 9, log, 1 << 27, 8 << 30)
    vx.reset_tuning()
    untuned = vx.tuning()  # knobs no sweep here times keep their defaults
    result = {
        "device": dev,
        "quick": bool(args.quick),
        "seconds": round(time.time() - t0, 1),
        "knobs": {**untuned, **sort_best, **scan_best, **edit_best, **small_best,
                  **serve_best},
        "timings_ms": {"sort": sort_t, "scan": scan_t, "edit": edit_t, "small": small_t,
                       "serve": serve_t},
    }
    out = args.out or str(tuning_file(dev))
    from pathlib import Path
    Path(out).parent.mkdir(parents=True, exist_ok=True)
    Path(out).write_text(json.dumps(result, indent=1) + "\n")
    log(f"best {result['knobs']} -> {out}")
    return result


if __name__ == "__main__":
    main()
