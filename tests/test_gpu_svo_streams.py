"""SVO edits beside other work on the GPU: a batched edit, a long voxel list
and a collection finish while a kernel of another stream (tests/hold_sm.cu)
has a multiprocessor to itself, and two worlds are edited on two streams at a time, against
the oracle."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu
LONG = 700_000_000  # ns that the other stream's kernel takes


@pytest.fixture(scope="module")
def hold_sm(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc is needed to build the other stream's kernel")
    out = tmp_path_factory.mktemp("hold") / "libhold.so"
    cmd = ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-shared",
           "-Xcompiler", "-fPIC", str(Path(__file__).with_name("hold_sm.cu")), "-o", str(out)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    fn = C.CDLL(str(out)).hold_sm
    fn.argtypes, fn.restype = [C.c_uint64, C.c_void_p], C.c_int
    return fn


def prims(rng, n, world):
    p = np.zeros(n, oracle.PRIM_DTYPE)
    p["c"] = rng.integers(0, world, (n, 3))
    p["r"][:, 0] = rng.integers(0, world // 8, n)
    op = rng.integers(0, 2, n)
    p["flags"] = (op << 8) | ((rng.integers(1, 4, n) * op) << 16)
    return p


def world_box(world, add):
    p = np.zeros(1, oracle.PRIM_DTYPE)
    p[0] = ((0, 0, 0), (world, world, world), 4 | (int(add) << 8) | (1 << 16), 0)
    return p


@pytest.mark.parametrize("what", ["batch", "list", "collect", "batch that collects"])
def test_finishes_beside_a_running_kernel(cuda, hold_sm, what):
    rng = np.random.default_rng(1)
    depth = 5
    world = 4 << depth
    p = prims(rng, 300, world)
    # "that collects": room for one such edit, whose remains the next reclaims
    room = 5000 if what == "batch that collects" else 1 << 18
    s = vx.Svo(depth, room, 8 * room, materials=True, arena_bytes=64 << 20)
    voxels = vx.voxels_to_device(rng.integers(0, world, (20000, 3)).astype(np.uint32), cuda)
    batch, fill = (vx.prims_to_device(x, cuda) for x in (p, world_box(world, True)))
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()

    def call():
        if what == "list":
            assert s.apply_voxels(voxels, 1) == 0
        elif what == "collect":
            s.collect()
        else:
            s.apply_primitives(batch)
            assert s.status() == 0

    torch.cuda.synchronize()
    with torch.cuda.stream(mine):
        for _ in range(3):  # kernels are loaded; subtrees are detached
            call()
            s.apply_primitives(fill)
            assert s.status() == 0
    mine.synchronize()
    assert hold_sm(1000, other.cuda_stream) == 0  # loaded
    other.synchronize()
    assert hold_sm(LONG, other.cuda_stream) == 0
    with torch.cuda.stream(mine):
        call()
    mine.synchronize()
    running = not other.query()
    other.synchronize()
    assert running, "the call waited for the other stream's kernel"
    if what.startswith("batch"):
        g = oracle.Grid(depth, materials=True).apply_prims(world_box(world, True)).apply_prims(p)
        assert oracle.SvoCanon(*s.canonical()) == g.svo()


def test_two_worlds_on_two_streams(cuda):
    """Batches on two worlds without a synchronisation in between, in room so
    small that edits collect (with the wait of one collection's blocks for
    one another beside the other's)."""
    rng = np.random.default_rng(2)
    depth = 5
    world = 4 << depth
    worlds = []
    for mats in (False, True):
        worlds.append((vx.Svo(depth, 5000, 40000, materials=mats, arena_bytes=64 << 20),
                       oracle.Grid(depth, materials=mats), torch.cuda.Stream()))
    edits = []
    for k in range(12):
        e = world_box(world, k % 4 == 1) if k % 2 else prims(rng, 300, world)
        edits.append((e, vx.prims_to_device(e, cuda)))
    torch.cuda.synchronize()
    for e, d in edits:
        for s, g, stream in worlds:
            with torch.cuda.stream(stream):
                s.apply_primitives(d)
            g.apply_prims(e)
    for s, g, stream in worlds:
        stream.synchronize()
        assert s.status() == 0
        assert oracle.SvoCanon(*s.canonical()) == g.svo()
