"""Ray casts whose exit side is hard to tell (equal, denormal, huge and tiny
direction components, origins on lattice planes) and counts on both sides of
a warp's and the device's share of rays, against the oracle's ray cast."""
import numpy as np
import pytest
import torch

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 400_003])
def test_edge_rays_match_oracle(cuda, n):
    depth = 6
    world = 4 << depth
    prims = vx.config_c4_edits(300, seed=12, world_exp=depth + 2)
    prims["r"] = np.minimum(prims["r"], world // 8)
    dag = vx.HashDag(depth, 1 << 20, 256 << 20)
    dag.build_terrain(5, 1, True)
    dag.apply_primitives(vx.prims_to_device(prims, cuda))
    assert dag.status() == 0
    rng = np.random.default_rng(n)
    r = np.zeros(n, vx.RAY_DTYPE)
    o = rng.uniform(-8, world + 8, (n, 3))
    lattice = rng.random(n) < 0.5
    o[lattice] = np.rint(o[lattice] * 2) / 2
    d = rng.normal(size=(n, 3))
    kind = rng.integers(0, 6, n)
    d[kind == 1] = np.sign(d[kind == 1])                      # exact diagonals
    d[kind == 2] = np.rint(d[kind == 2] * 2)                  # small integers, zeros
    for k, scale in ((3, 1e-40), (4, 1e-30), (5, 1e30)):      # one odd component
        rows = np.flatnonzero(kind == k)
        d[rows, rng.integers(0, 3, len(rows))] *= scale
    r["origin"], r["dir"] = o, d
    r["t_max"] = np.where(rng.random(n) < 0.2, rng.uniform(0, world, n), 3.0e38)
    got = dag.raycast(torch.from_numpy(r.view(np.uint8)).to(cuda)).cpu().numpy()
    want = oracle.Sparse(depth, oracle.terrain(5, 1, True), prims).raycast(r)
    assert np.array_equal(got.view(np.uint32).reshape(-1, 5), want)
