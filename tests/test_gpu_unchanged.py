"""Edits whose primitives leave part of the world as it is (added to solid
ground, removed from air, one material over the same material) beside ones
that change it, on terrain and on uniform worlds, in batches for each of the
expansion's list lengths and as voxel lists, against the oracle."""
import numpy as np
import pytest

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu


def prims(rng, n, world, kind):
    p = np.zeros(n, oracle.PRIM_DTYPE)
    shape = rng.integers(0, 2, n)
    p["c"] = rng.integers(0, world, (n, 3))
    r = rng.integers(0, world // 6, (n, 3))
    p["r"] = np.where(shape[:, None] == 1, r, r * [1, 0, 0])
    op = {"add": np.ones(n, int), "remove": np.zeros(n, int)}.get(kind, rng.integers(0, 2, n))
    mat = rng.integers(1, 3, n)  # few materials: many meet their own
    p["flags"] = shape | (op << 8) | ((mat * op) << 16)
    return p


@pytest.mark.parametrize("kind", ["add", "remove", "both"])
@pytest.mark.parametrize("n", [1, 40, 300, 3000])
@pytest.mark.parametrize("start", ["terrain", "empty", "full"])
def test_batches(cuda, kind, n, start):
    rng = np.random.default_rng(n + len(kind))
    depth = 5
    world = 4 << depth
    t = oracle.terrain(seed=3, scale=1, caves=True)
    box = np.zeros(1, oracle.PRIM_DTYPE)
    box[0] = ((0, 0, 0), (world, world, world), 4 | (1 << 8) | (1 << 16), 0)
    p = prims(rng, n, world, kind)
    cases = [(vx.HashDag(depth, 1 << 18, 64 << 20), False)]
    cases += [(vx.Svo(depth, 1 << 18, 1 << 18, materials=m, arena_bytes=64 << 20), m)
              for m in (False, True)]
    for s, mats in cases:
        g = oracle.Grid(depth, materials=mats)
        if start == "terrain":
            s.build_terrain(3, 1, True)
            g.terrain(t)
        elif start == "full":
            s.apply_primitives(vx.prims_to_device(box, cuda))
            g.apply_prims(box)
        s.apply_primitives(vx.prims_to_device(p, cuda))
        assert s.status() == 0
        g.apply_prims(p)
        if isinstance(s, vx.HashDag):
            assert oracle.DagCanon(*s.canonical()) == g.dag()
        else:
            assert oracle.SvoCanon(*s.canonical()) == g.svo()


@pytest.mark.parametrize("n", [500, 20000])
def test_voxel_lists_on_terrain(cuda, n):
    rng = np.random.default_rng(n)
    depth = 5
    dag, g = vx.HashDag(depth, 1 << 18, 64 << 20), oracle.Grid(depth)
    dag.build_terrain(3, 1, True)
    g.terrain(oracle.terrain(seed=3, scale=1, caves=True))
    for op in (1, 0, 1):
        v = rng.integers(0, 4 << depth, (n, 3)).astype(np.uint32)
        assert dag.apply_voxels(vx.voxels_to_device(v, cuda), op) == 0
        g.apply_voxels(v, op)
        assert oracle.DagCanon(*dag.canonical()) == g.dag()
