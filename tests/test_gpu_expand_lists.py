"""Batched expansion around its list lengths: items with one primitive, with a
few (up to 32 and beyond), long lists on one block and on a cluster of blocks
(4,096), lists past a block's kept bits, mixed shapes, against the oracle."""
import numpy as np
import pytest

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu


def prims(kind, n, world, rng):
    p = np.zeros(n, oracle.PRIM_DTYPE)
    shape = rng.integers(0, 2, n) if kind != "spheres" else np.zeros(n, int)
    p["c"] = rng.integers(-2, world + 2, (n, 3))
    r = rng.integers(0, 4, (n, 3))
    r[rng.random(n) < 0.02] += world // 8  # a few that cover whole cells
    if kind == "stack":  # all on one spot: one leaf parent holds every primitive
        p["c"] = world // 2 + rng.integers(0, 6, (n, 3))
    p["r"] = np.where(shape[:, None] == 1, r, r * [1, 0, 0])
    op = (rng.random(n) < 0.55).astype(np.uint32)
    p["flags"] = shape | (op << 8) | (rng.integers(1, 256, n) * op) << 16
    return p


@pytest.mark.parametrize("kind", ["spheres", "mixed", "stack"])
@pytest.mark.parametrize("n", [257, 4096, 4097, 33000, 70001])
def test_list_lengths_match_oracle(cuda, kind, n):
    if kind == "stack":
        n = min(n, 4097)  # every primitive meets every touched leaf
    rng = np.random.default_rng(n)
    depth = 5
    p = prims(kind, n, 4 << depth, rng)
    d = vx.prims_to_device(p, cuda)
    dag = vx.HashDag(depth, 1 << 18, 256 << 20)
    dag.apply_primitives(d)
    assert dag.status() == 0
    g = oracle.Grid(depth).apply_prims(p)
    assert oracle.DagCanon(*dag.canonical()) == g.dag()
    for mats in (False, True):
        svo = vx.Svo(depth, 1 << 18, 1 << 18, materials=mats, arena_bytes=256 << 20)
        svo.apply_primitives(d)
        assert svo.status() == 0
        assert (oracle.SvoCanon(*svo.canonical())
                == oracle.Grid(depth, materials=mats).apply_prims(p).svo())


def test_failed_edit_leaves_every_cluster(cuda):
    """An arena too small for a batch with cluster-expanded lists: reported,
    old content kept."""
    depth = 5
    rng = np.random.default_rng(3)
    dag = vx.HashDag(depth, 1 << 16, 1 << 20)
    before = oracle.DagCanon(*dag.canonical())
    dag.apply_primitives(vx.prims_to_device(prims("mixed", 50000, 4 << depth, rng), cuda))
    assert dag.status() == vx.VX_ERR_CAPACITY
    assert oracle.DagCanon(*dag.canonical()) == before
