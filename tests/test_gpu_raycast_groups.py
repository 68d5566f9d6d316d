"""Ray lists on both sides of the length from which groups of 32 like rays and
the others go to different kernels: groups from one eye, parallel groups, groups
with one odd ray, random ones, rays that are no rays, a short last group;
against the oracle's ray cast, with every hit written."""
import numpy as np
import pytest
import torch

import oracle
import voxel_b200 as vx

pytestmark = pytest.mark.gpu
FEWEST = 3 << 17


def grouped_rays(rng, n, world):
    g = (n + 31) // 32
    kind = np.repeat(rng.integers(0, 5, g), 32)[:n]
    o, d = rng.uniform(0, world, (n, 3)), rng.normal(size=(n, 3))
    eye = np.repeat(rng.uniform(0, world, (g, 3)), 32, 0)[:n]
    look = np.repeat(rng.normal(size=(g, 3)), 32, 0)[:n]
    spread = np.repeat(rng.choice([0.0, 0.02, 0.2, 0.5], g), 32)[:n, None]
    one = kind != 0  # 0: random
    o[one] = eye[one]
    d[one] = (look + spread * rng.normal(size=(n, 3)))[one]
    par = kind == 2
    o[par] += rng.uniform(-world / 12, world / 12, (par.sum(), 3))
    d[par] = look[par]
    odd = (kind == 3) & (rng.random(n) < 1 / 32)
    d[odd] *= -1
    none = (kind == 4) & (rng.random(n) < 1 / 16)
    d[none] = rng.choice([0.0, np.nan, np.inf], (none.sum(), 3))
    r = np.zeros(n, vx.RAY_DTYPE)
    r["origin"], r["dir"] = o, d
    r["t_max"] = np.where(rng.random(n) < 0.1, rng.uniform(0, world, n), 3.0e38)
    return r


@pytest.mark.parametrize("n", [31, FEWEST, FEWEST + 1, FEWEST + 32, 500_001])
def test_grouped_rays_match_oracle(cuda, n):
    depth = 6
    world = 4 << depth
    prims = vx.config_c4_edits(200, seed=13, world_exp=depth + 2)
    prims["r"] = np.minimum(prims["r"], world // 8)
    dag = vx.HashDag(depth, 1 << 20, 256 << 20)
    dag.build_terrain(5, 1, True)
    dag.apply_primitives(vx.prims_to_device(prims, cuda))
    assert dag.status() == 0
    r = grouped_rays(np.random.default_rng(n), n, world)
    d_rays = torch.from_numpy(r.view(np.uint8)).to(cuda)
    dag.raycast(torch.zeros_like(d_rays))  # (what the allocator hands out next is no result)
    got = dag.raycast(d_rays).cpu().numpy().view(np.uint32).reshape(-1, 5)
    want = oracle.Sparse(depth, oracle.terrain(5, 1, True), prims).raycast(r)
    # a NaN has no voxel that the oracle would name: as in a short list
    nan = np.isnan(r["dir"]).any(1)
    if nan.any():
        alone = dag.raycast(torch.from_numpy(r[nan].view(np.uint8)).to(cuda))
        want[nan] = alone.cpu().numpy().view(np.uint32).reshape(-1, 5)
    assert np.array_equal(got, want)
