"""Scans around the one-block limit (64 KB), the edges of tiles and of groups of
32 tiles, and more groups than one look-back reads, against numpy."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx

pytestmark = pytest.mark.gpu

TILE = {4: 8192, 8: 4096}  # elements of the default 32 KB tile
SMALL = {4: 16384, 8: 8192}


@pytest.mark.parametrize("each", [4, 8])
@pytest.mark.parametrize("shift", [0, 1])  # 16-byte aligned or not
def test_sizes_around_every_edge(cuda, each, shift):
    t, s = TILE[each], SMALL[each]
    sizes = [1, 3, 4, 5, 127, 128, 4097, s - 1, s, s + 1, 3 * t - 1, 3 * t, 3 * t + 1,
             32 * t - 1, 32 * t, 32 * t + 1, 33 * t, 64 * t + 7, 1025 * t + 3]
    dt = np.uint32 if each == 4 else np.uint64
    rng = np.random.default_rng(each + shift)
    x = rng.integers(0, np.iinfo(dt).max, max(sizes) + 1, dtype=dt, endpoint=True)
    x[: 40 * t] = np.iinfo(dt).max  # the largest sums a group can hold
    signed = np.int32 if each == 4 else np.int64
    for n in sizes:
        d = torch.from_numpy(x.view(signed)).to(cuda)[shift:shift + n]
        ws = torch.full((vx.lib().vx_scan_workspace_size(n),), 0x5A, dtype=torch.uint8,
                        device=cuda)
        total = np.cumsum(x[shift:shift + n], dtype=dt)
        want = np.concatenate([np.zeros(1, dt), total[:-1]])
        vx.exclusive_sum(d, ws)
        assert vx.workspace_status(ws) == 0
        assert np.array_equal(d.cpu().numpy().view(dt), want), n
        if each == 4:
            d = torch.from_numpy(x.view(signed)).to(cuda)[shift:shift + n]
            vx.inclusive_sum(d, ws)
            assert np.array_equal(d.cpu().numpy().view(dt), total), n
