"""What a user of this library has it do, as measurable cases.

Each case is one path of the public API at one size; draw() gives more cases
of the same paths with sizes spread over the ranges that RANGES declares.
prepare() makes what a program holds before the call (structures, inputs,
workspaces), run() is one pass through the public entry points.

Every pass can be repeated on its state: sorts start from a kept unsorted
copy, batched Hash DAG edits from a kept snapshot (vx_dag_copy), table fills
from a cleared table, and the other edits come in pairs whose second undoes
or overwrites what the first did, so that each pass does the same work.
"""
import math

import numpy as np
import torch

import voxel_b200 as vx

DEVICE = "cuda"
ADD, REMOVE = 1, 0
HASH_LOAD = 0.8  # as in the benchmark's hash tables

# Smallest and largest size of each kind (elements, keys, primitives, voxels'
# sphere radius, rays), as the benchmark, the tests and the served stream use.
RANGES = {
    "scan": (10007, 1 << 27),
    "sort": (1 << 16, 1 << 26),
    "slab": (1 << 18, 1 << 24),
    "cuckoo": (1 << 18, 1 << 24),
    "strokes": (2, 16),
    "voxels": (24, 128),
    "svo_batch": (512, 65536),
    "undo": (1, 256),
    "dag_batch": (512, 16384),
    "raycast": (1 << 16, 1 << 20),
}


def listed():
    return [
        # The smallest call of the primitives: an allocator's or a frame
        # loop's offsets, one allocation of scratch and one scan.
        {"name": "scan_u32_small", "kind": "scan", "n": 10007, "bytes_each": 4},
        # Offsets of a large stream compaction (the benchmark's scan scaled to
        # half its size, with a ragged end).
        {"name": "scan_u32_large", "kind": "scan", "n": (1 << 27) + 5, "bytes_each": 4},
        # Ordering a mid-sized edit list by a 32-bit key with its index.
        {"name": "sort_u32_mid", "kind": "sort", "n": (1 << 20) + 7, "bytes_each": 4, "bits": 32},
        # Ordering points by 60-bit Morton codes with their index: the
        # benchmark's Morton sort at a quarter of its size.
        {"name": "sort_u64_morton_large", "kind": "sort", "n": 1 << 26, "bytes_each": 8, "bits": 60},
        # Filling a slab set to load 0.8 and probing it at 50 % hits.
        {"name": "slab_set", "kind": "slab", "n": 1 << 24},
        # The same for the cuckoo map, at a size whose table is near L2's.
        {"name": "cuckoo_map", "kind": "cuckoo", "n": (1 << 22) + 1},
        # Interactive brush strokes: four plain calls of a few thousand voxels
        # on a 256^3 SVO with materials, then a look at the result.
        {"name": "svo_strokes", "kind": "strokes", "radius": 10},
        # The reference's published voxel edit: a sphere of 8.78 M voxels as
        # a voxel list, placed in and removed from a 4096^3 SVO.
        {"name": "svo_voxels_sphere", "kind": "voxels", "store": "svo", "radius": 128},
        # Batched mixed spheres and boxes on a 4096^3 SVO with materials.
        {"name": "svo_batch", "kind": "svo_batch", "n": 65536},
        # An editor's do and undo of one small request (the served stream's
        # size) on a resident 2048^3 Hash DAG.
        {"name": "dag_undo", "kind": "undo", "n": 32},
        # The headline: 16,384 spheres on a 16384^3 Hash DAG, from a snapshot.
        {"name": "dag_batch_large", "kind": "dag_batch", "n": 16384, "depth": 12},
        # One frame of primary and random rays on a 4096^3 Hash DAG.
        {"name": "dag_raycast", "kind": "raycast", "n": 1 << 20},
    ]


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    lo, hi = RANGES[kind]
    size = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "scan":
        each = rng.choice((4, 8))
        return {"kind": kind, "n": max(lo, size * 4 // each) | 1, "bytes_each": each}
    if kind == "sort":
        each = rng.choice((4, 8))
        bits = rng.choice((32, 24, 17)) if each == 4 else rng.choice((60, 64, 37))
        return {"kind": kind, "n": size, "bytes_each": each, "bits": bits}
    if kind in ("strokes", "voxels"):
        case = {"kind": kind, "radius": size}
        if kind == "voxels":
            case["store"] = rng.choice(("svo", "dag"))
        case["shift"] = rng.randrange(1 << 16)  # where in the world
        return case
    if kind == "dag_batch":
        return {"kind": kind, "n": size, "depth": rng.choice((9, 10))}
    return {"kind": kind, "n": size}


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _ints(n, bits, each, seed):
    """n random keys of `bits` bits in int32 / int64."""
    g = _generator(seed)
    if each == 4:
        lo, hi = (-(1 << 31), (1 << 31)) if bits == 32 else (0, 1 << bits)
        return torch.randint(lo, hi, (n,), dtype=torch.int64, device=DEVICE,
                             generator=g).to(torch.int32)
    lo, hi = (-(1 << 63), (1 << 63) - 1) if bits == 64 else (0, 1 << bits)
    return torch.randint(lo, hi, (n,), dtype=torch.int64, device=DEVICE, generator=g)


def _spread3(x):
    """Bits 0-19 of x moved to every third bit."""
    x = (x | (x << 32)) & 0x1F00000000FFFF
    x = (x | (x << 16)) & 0x1F0000FF0000FF
    x = (x | (x << 8)) & 0x100F00F00F00F00F
    x = (x | (x << 4)) & 0x10C30C30C30C30C3
    return (x | (x << 2)) & 0x1249249249249249


def _keys(case, seed):
    if case["bytes_each"] == 8 and case["bits"] == 60:  # Morton codes of points in a 2^20 cube
        g = _generator(seed)
        code = None
        for a in range(3):
            c = _spread3(torch.randint(0, 1 << 20, (case["n"],), dtype=torch.int64,
                                       device=DEVICE, generator=g)) << a
            code = c if code is None else code | c
        return code
    return _ints(case["n"], case["bits"], case["bytes_each"], seed)


def _hash_keys(n, seed):
    """n keys to insert and n to look up, half of those present."""
    g = _generator(seed)
    keys = torch.randint(-2**63, 2**63 - 2, (n,), dtype=torch.int64, device=DEVICE, generator=g)
    probe = torch.randint(-2**63, 2**63 - 2, (n,), dtype=torch.int64, device=DEVICE, generator=g)
    probe[: n // 2] = keys[torch.randint(0, n, (n // 2,), device=DEVICE, generator=g)]
    return keys, probe[torch.randperm(n, device=DEVICE, generator=g)].contiguous()


def _points(n, world, prims, seed):
    """n voxels of the world: half anywhere, half within a primitive's box."""
    g = np.random.default_rng(seed)
    p = g.integers(0, world, (n, 3))
    which = g.integers(0, len(prims), n // 2)
    c = prims["c"][which].astype(np.int64)
    r = prims["r"][which].astype(np.int64)
    r = np.where(r == 0, r[:, :1], r)  # a sphere has its radius in the first
    p[: n // 2] = np.clip(c + np.rint(g.uniform(-1.2, 1.2, c.shape) * r), 0, world - 1)
    return vx.voxels_to_device(p.astype(np.uint32), DEVICE)


def _rays(n, world, seed):
    g = np.random.default_rng(seed)
    r = np.zeros(n, vx.RAY_DTYPE)
    o = g.uniform(0, world, (n, 3))
    down = g.random(n) < 0.5
    o[down, 2] = g.uniform(world * 0.62, world * 0.75, int(down.sum()))
    d = g.normal(size=(n, 3))
    d[down, 2] = -np.abs(d[down, 2]) - 0.3
    r["origin"], r["dir"], r["t_max"] = o, d, 3.0e38
    return vx.records_to_device(r, DEVICE)


def _ok(status):
    if status != 0:
        raise RuntimeError(f"edit failed with status {status}")


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "scan":
        each = case["bytes_each"]
        s["data"] = _ints(case["n"], 32 if each == 4 else 64, each, seed)
        if case["n"] > 1 << 16:  # a small caller lets the call take its scratch
            s["ws"] = torch.empty(vx.lib().vx_scan_workspace_size(case["n"]), dtype=torch.uint8,
                                  device=DEVICE)
    elif kind == "sort":
        s["src"] = _keys(case, seed)
        s["index"] = torch.arange(case["n"], dtype=torch.int32, device=DEVICE)
        s["keys"], s["values"] = torch.empty_like(s["src"]), torch.empty_like(s["index"])
        s["bits"] = case["bits"]
        s["ws"] = torch.empty(vx.lib().vx_sort_workspace_size(case["n"], case["bytes_each"]),
                              dtype=torch.uint8, device=DEVICE)
    elif kind in ("slab", "cuckoo"):
        n = case["n"]
        s["keys"], s["probe"] = _hash_keys(n, seed)
        s["status"] = torch.empty(n, dtype=torch.int32, device=DEVICE)
        if kind == "slab":
            s["table"] = vx.SlabHashSet(int(n / (HASH_LOAD * 15)) + 1, n // 30)
        else:
            s["table"] = vx.CuckooMap(int(n / HASH_LOAD) + 1, 2000)
    elif kind == "strokes":
        svo = vx.Svo(6, 1 << 18, 1 << 18, materials=True, arena_bytes=64 << 20)
        svo.build_terrain(1, 1, False)
        _ok(svo.status())
        r = case["radius"]
        prims = vx.generate_primitives(8, 4, seed + case.get("shift", 0), r_min=max(1, r - 1),
                                       r_max=r + 1)
        vox, off = vx.rasterize(vx.prims_to_device(prims, DEVICE), 8)
        off = off.cpu().tolist()
        s["svo"] = svo
        s["calls"] = [(vox[off[i]:off[i + 1]], (ADD, REMOVE, ADD, REMOVE)[i], 1 + (seed + i) % 255)
                      for i in range(4)]
        most = max(off[i + 1] - off[i] for i in range(4))
        s["ws"] = torch.empty(vx.lib().vx_svo_voxel_workspace_size(most), dtype=torch.uint8,
                              device=DEVICE)
        s["points"] = _points(1 << 16, 256, prims, seed)
    elif kind == "voxels":
        r, world = case["radius"], 4096
        g = np.random.default_rng(seed + case.get("shift", 0))
        prim = np.zeros(1, vx.PRIM_DTYPE)
        prim["c"][0] = g.integers(r, world - r, 3)
        prim["r"][0, 0] = r
        prim["flags"] = vx.make_flags(0, ADD)
        s["voxels"], _ = vx.rasterize(vx.prims_to_device(prim, DEVICE), 12)
        n = s["voxels"].shape[0]
        # the list in a mixed order, as threads of a tool would emit it
        s["voxels"] = s["voxels"][torch.randperm(n, device=DEVICE, generator=_generator(seed))]
        s["voxels"] = s["voxels"].contiguous()
        if case["store"] == "svo":
            s["world"] = vx.Svo(10, 1 << 21, 1 << 21, arena_bytes=1 << 30)
            size = vx.lib().vx_svo_voxel_workspace_size(n)
        else:
            s["world"] = vx.HashDag(10, 1 << 22, 1 << 30)
            s["world"].build_terrain(6, 16, True)
            _ok(s["world"].status())
            size = s["world"].workspace_size(n)
        s["ws"] = torch.empty(size, dtype=torch.uint8, device=DEVICE)
        s["points"] = _points(1 << 18, world, prim, seed)
    elif kind == "svo_batch":
        n = case["n"]
        svo = vx.Svo(10, 1 << 24, 1 << 26, materials=True, arena_bytes=2 << 30)
        svo.build_terrain(6, 16, True)
        _ok(svo.status())
        prims = vx.config_c3_edits(n, seed=seed)
        s["svo"] = svo
        s["halves"] = [vx.prims_to_device(prims[: n // 2], DEVICE),
                       vx.prims_to_device(prims[n // 2:], DEVICE)]
        s["points"] = _points(1 << 20, 4096, prims, seed)
    elif kind == "undo":
        dag = vx.HashDag(9, 1 << 22, 512 << 20)
        dag.build_terrain(7, 8, True)
        _ok(dag.status())
        do = vx.generate_primitives(11, case["n"], seed, sphere_permille=500, r_min=1, r_max=128,
                                    log_uniform=True)
        undo = do.copy()
        undo["flags"] ^= 1 << 8  # the opposite operation
        s["dag"] = dag
        s["do"], s["undo"] = vx.prims_to_device(do, DEVICE), vx.prims_to_device(undo, DEVICE)
        s["points"] = _points(1 << 16, 2048, do, seed)
    elif kind == "dag_batch":
        n, depth = case["n"], case["depth"]
        most = 1 << 25 if depth == 12 else 1 << 23
        s["base"] = vx.HashDag(depth, most, 6 << 30 if depth == 12 else 1 << 30)
        s["base"].build_terrain(7, 1 << (depth - 6), True)
        _ok(s["base"].status())
        s["dag"] = vx.HashDag(depth, most, 4 << 30 if depth == 12 else 2 << 30)
        world = 4 << depth
        prims = vx.config_c4_edits(n, seed=seed, world_exp=depth + 2) if depth == 12 else \
            vx.generate_primitives(depth + 2, min(n, 4096), seed, add_permille=600, r_min=1,
                                   r_max=256 if depth == 10 else 128, log_uniform=True)
        s["prims"] = vx.prims_to_device(prims, DEVICE)
        # the edited window that is read back for meshing: 1024 x 1024 x 64
        # voxels around the largest sphere
        c = prims["c"][int(prims["r"][:, 0].argmax())].astype(np.int64) // 4
        size = (256, 256, 16)
        s["lo"] = [int(min(max(0, c[a] - size[a] // 2), world // 4 - size[a])) for a in range(3)]
        s["size"] = size
        s["points"] = _points(1 << 18, world, prims, seed)
    elif kind == "raycast":
        s["dag"] = vx.HashDag(10, 1 << 22, 1 << 30)
        s["dag"].build_terrain(6, 16, True)
        _ok(s["dag"].status())
        s["rays"] = _rays(case["n"], 4096, seed)
    return s


def run(s):
    kind = s["kind"]
    if kind == "scan":
        return vx.exclusive_sum(s["data"], s.get("ws"))
    if kind == "sort":
        s["keys"].copy_(s["src"])
        s["values"].copy_(s["index"])
        return vx.sort_pairs(s["keys"], s["values"], s["bits"], s["ws"])
    if kind == "slab":
        s["table"].clear()
        s["table"].insert(s["keys"], s["status"])
        return s["status"], s["table"].contains(s["probe"])
    if kind == "cuckoo":
        s["table"].clear()
        s["table"].insert(s["keys"], None, s["status"])
        return s["status"], s["table"].find(s["probe"])
    if kind == "strokes":
        for vox, op, material in s["calls"]:
            _ok(s["svo"].apply_voxels(vox, op, material, s["ws"]))
        return s["svo"].query(s["points"])
    if kind == "voxels":
        w = s["world"]
        extra = (1,) if isinstance(w, vx.Svo) else ()
        _ok(w.apply_voxels(s["voxels"], ADD, *extra, workspace=s["ws"]))
        placed = w.query(s["points"])
        _ok(w.apply_voxels(s["voxels"], REMOVE, *extra, workspace=s["ws"]))
        return placed, w.query(s["points"])
    if kind == "svo_batch":
        for half in s["halves"]:
            s["svo"].apply_primitives(half)
        _ok(s["svo"].status())
        return s["svo"].query(s["points"])
    if kind == "undo":
        s["dag"].apply_primitives(s["do"])
        _ok(s["dag"].status())
        done = s["dag"].query(s["points"])
        s["dag"].apply_primitives(s["undo"])
        _ok(s["dag"].status())
        return done, s["dag"].query(s["points"])
    if kind == "dag_batch":
        s["dag"].copy_from(s["base"])
        s["dag"].apply_primitives(s["prims"])
        _ok(s["dag"].status())
        return s["dag"].read_leaves(s["lo"], s["size"]), s["dag"].query(s["points"])
    return s["dag"].raycast(s["rays"])


def _sphere_voxels(r):
    return 4.18879 * (r + 0.5) ** 3


def _surface_cells(r_min, r_max):
    """8^3 cells that the surface of a sphere with a log-uniform radius cuts,
    on average."""
    mean_r2 = (r_max ** 2 - r_min ** 2) / (2 * math.log(r_max / r_min))
    return max(1.0, 1.5 * 4 * math.pi * mean_r2 / 64)


def work(case):
    """Inputs once, outputs once, and of a structure the entries that change:
    16 bytes a hash entry, a leaf's mask and materials, and 56 bytes a changed
    Hash DAG node (the old item, the new one, its index entry)."""
    kind, n = case["kind"], case.get("n", 0)
    if kind == "scan":
        b = 2 * n * case["bytes_each"]
    elif kind == "sort":
        b = 2 * n * (case["bytes_each"] + 4)
    elif kind in ("slab", "cuckoo"):
        b = n * (8 + 4 + 16) + n * (8 + 4 + 16)
    elif kind == "strokes":
        v = _sphere_voxels(case["radius"])
        b = 4 * (12 * v + v / 64 * 2 * 72) + (1 << 16) * 13
    elif kind == "voxels":
        v = _sphere_voxels(case["radius"])
        b = 2 * (12 * v + v / 64 * 16) + 2 * (1 << 18) * 13
    elif kind == "svo_batch":
        b = n * (32 + _surface_cells(1, 64) * 4 * 2 * 72) + (1 << 20) * 13
    elif kind == "undo":
        b = 2 * n * (32 + _surface_cells(1, 128) * 56) + 2 * (1 << 16) * 13
    elif kind == "dag_batch":
        count = n if case["depth"] == 12 else min(n, 4096)
        b = count * (32 + _surface_cells(1, 128 if case["depth"] == 9 else 256) * 56)
        b += (1 << 20) * 8 + (1 << 18) * 13
    else:
        b = n * (32 + 20)
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """The primitives' and tables' results by torch alone."""
    kind = case["kind"]
    if kind == "scan":
        x = _ints(case["n"], 32 if case["bytes_each"] == 4 else 64, case["bytes_each"], seed)
        total = torch.cumsum(x, 0, dtype=torch.int64)  # wraps modulo 2^64
        out = torch.zeros_like(total)
        out[1:] = total[:-1]
        return out.to(x.dtype) if case["bytes_each"] == 8 else \
            ((out + (1 << 31)) % (1 << 32) - (1 << 31)).to(torch.int32)
    if kind == "sort":
        keys = _keys(case, seed)
        order = (keys ^ torch.iinfo(keys.dtype).min) if case["bits"] == 8 * case["bytes_each"] \
            else keys
        index = torch.sort(order, stable=True).indices
        return keys[index], index.to(torch.int32)
    return None
