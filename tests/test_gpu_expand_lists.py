"""Batched expansion around its list lengths: items with one primitive, with a
few (up to 32 and beyond), long lists on one block and on a cluster of blocks
(4,096), lists past the bits that a cluster keeps (262,144), mixed shapes, on
both sides of the level size from which a lane takes an item, against the
oracle."""
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


@pytest.mark.parametrize("kind", ["spheres", "mixed"])
def test_a_list_past_the_kept_bits_matches_oracle(cuda, kind):
    n = 270_001  # 8 blocks keep 32,768 primitives' bits each
    rng = np.random.default_rng(n)
    depth = 5
    p = prims(kind, n, 4 << depth, rng)
    p["r"][rng.random(n) < 0.9] = 0  # mostly single voxels: the oracle applies all of them
    d = vx.prims_to_device(p, cuda)
    dag = vx.HashDag(depth, 1 << 18, 512 << 20)
    dag.apply_primitives(d)
    assert dag.status() == 0
    svo = vx.Svo(depth, 1 << 18, 1 << 18, materials=True, arena_bytes=512 << 20)
    svo.apply_primitives(d)
    assert svo.status() == 0
    assert oracle.DagCanon(*dag.canonical()) == oracle.Grid(depth).apply_prims(p).dag()
    assert (oracle.SvoCanon(*svo.canonical())
            == oracle.Grid(depth, materials=True).apply_prims(p).svo())


@pytest.mark.parametrize("n", [300, 12000])
@pytest.mark.parametrize("boxes", [False, True])
def test_levels_of_few_and_many_items_match_oracle(cuda, n, boxes):
    """A crowd (few items, several primitives each) and primitives all over
    the world (levels of more than 37,888 items) on a 512^3 world."""
    depth = 7
    world = 4 << depth
    rng = np.random.default_rng(n + boxes)
    p = np.zeros(n, oracle.PRIM_DTYPE)
    if n == 300:
        p["c"] = world // 2 + rng.integers(-32, 32, (n, 3))
        r = rng.integers(4, 28, (n, 3))
    else:
        p["c"] = rng.integers(0, world, (n, 3))
        r = rng.integers(2, 9, (n, 3))
    p["r"] = r if boxes else r * [1, 0, 0]
    op = rng.integers(0, 2, n)
    p["flags"] = int(boxes) | (op << 8) | ((rng.integers(1, 4, n) * op) << 16)
    d = vx.prims_to_device(p, cuda)
    dag = vx.HashDag(depth, 1 << 21, 1 << 30)
    dag.build_terrain(3, 2, True)
    dag.apply_primitives(d)
    assert dag.status() == 0
    t = oracle.terrain(seed=3, scale=2, caves=True)
    assert (oracle.DagCanon(*dag.canonical())
            == oracle.Grid(depth).terrain(t).apply_prims(p).dag())
    svo = vx.Svo(depth, 1 << 20, 1 << 22, materials=True, arena_bytes=1 << 30)
    svo.build_terrain(3, 2, True)
    svo.apply_primitives(d)
    assert svo.status() == 0
    assert (oracle.SvoCanon(*svo.canonical())
            == oracle.Grid(depth, materials=True).terrain(t).apply_prims(p).svo())


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
