"""Long voxel and leaf-command lists (sorted, reduced to leaf masks and expanded
by key ranges) against the oracle, and against the same list in chunks short
enough for the single cooperative launch, which neither sorts nor searches."""
import numpy as np
import pytest

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu

CHUNK = 16384  # the longest list of the cooperative path


def voxel_list(kind, n, world, rng):
    v = rng.integers(0, world, (n, 3))
    if kind == "one":  # a single run across many warps
        v[:] = v[0]
    elif kind == "runs":  # runs of every length around a warp's
        v = np.repeat(v[: n // 33 + 1], rng.integers(1, 70, n // 33 + 1), axis=0)[:n]
        v = np.concatenate([v, rng.integers(0, world, (n - len(v), 3))])
    elif kind == "dense":  # whole leaves and their neighbours
        side = int(np.ceil(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        v = (g + rng.integers(0, max(1, world - side), 3)) % world
    elif kind == "outside":
        v[::2] += world
    elif kind == "none":
        v += world
    return v[rng.permutation(len(v))].astype(np.uint32)


@pytest.mark.parametrize("kind", ["random", "one", "runs", "dense", "outside", "none"])
@pytest.mark.parametrize("depth,n", [(1, 16385), (4, 20011), (10, 40001), (11, 40001)])
def test_long_lists_equal_oracle_and_short_lists(cuda, kind, depth, n):
    rng = np.random.default_rng(depth * 100 + n)
    world = 4 << depth
    place, destroy = (voxel_list(kind, n, world, rng) for _ in range(2))
    destroy = np.concatenate([destroy, place[: n // 2]])
    for make in (lambda: vx.HashDag(depth, 1 << 20, 256 << 20),
                 lambda: vx.Svo(depth, 1 << 20, 1 << 20, arena_bytes=256 << 20)):
        long, short = make(), make()
        for v, op in ((place, vx.EDIT_PLACE), (destroy, vx.EDIT_DESTROY)):
            assert long.apply_voxels(vx.voxels_to_device(v, cuda), op) == 0
            for i in range(0, len(v), CHUNK):
                assert short.apply_voxels(vx.voxels_to_device(v[i:i + CHUNK], cuda), op) == 0
            canon = oracle.DagCanon if isinstance(long, vx.HashDag) else oracle.SvoCanon
            assert canon(*long.canonical()) == canon(*short.canonical())
            if depth <= 4:
                g = oracle.Grid(depth).apply_voxels(place, 1)
                if op == vx.EDIT_DESTROY:
                    g.apply_voxels(destroy, 0)
                want = g.dag() if isinstance(long, vx.HashDag) else g.svo()
                assert canon(*long.canonical()) == want


@pytest.mark.parametrize("depth", [2, 10, 11])
def test_long_command_lists_equal_short_ones(cuda, depth):
    rng = np.random.default_rng(depth)
    n = 20001
    c = np.zeros(n, vx.LEAF_COMMAND_DTYPE)
    for a in ("leaf_x", "leaf_y", "leaf_z"):
        c[a] = rng.integers(0, (1 << depth) + 1, n)  # some outside
    c[n // 2:] = c[rng.integers(0, n // 2, n - n // 2)]
    for a in ("voxel_data_low", "voxel_data_high"):
        c[a] = rng.integers(0, 1 << 32, n, dtype=np.uint64)
    long, short = (vx.HashDag(depth, 1 << 20, 256 << 20) for _ in range(2))
    assert long.apply_leaf_commands(vx.records_to_device(c, cuda), vx.EDIT_PLACE) == 0
    for i in range(0, n, CHUNK):
        assert short.apply_leaf_commands(vx.records_to_device(c[i:i + CHUNK], cuda),
                                         vx.EDIT_PLACE) == 0
    assert oracle.DagCanon(*long.canonical()) == oracle.DagCanon(*short.canonical())
