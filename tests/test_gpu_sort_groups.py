"""Sorts whose tile counts lie around groups of 8 and super-groups of 64 tiles
and reach past the super-groups of one look-back round, with digits that all
keys share and digits that none has, against a stable argsort."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("each", [4, 8])
@pytest.mark.parametrize("items", ["small", "large"])
def test_tile_counts_around_every_group(cuda, each, items):
    knob = f"sort.items_u{8 * each}"
    per = vx.tuning_options(knob)[0 if items == "small" else 1]
    tile = 256 * per
    dt, signed = (np.uint32, np.int32) if each == 4 else (np.uint64, np.int64)
    rng = np.random.default_rng(each * per)
    try:
        vx.set_tuning(knob, per)
        for tiles in (1, 7, 8, 9, 63, 64, 65, 128, 129, 400, 513):
            for n in (tile * tiles - 1, tile * tiles, tile * tiles + 1):
                k = rng.integers(0, np.iinfo(dt).max, n, dtype=dt, endpoint=True)
                k &= dt(0xFF0000FF)      # two digits the same for all
                k[rng.random(n) < 0.7] = dt(0x55000033)  # one heavy key
                d = torch.from_numpy(k.view(signed)).to(cuda)
                v = torch.arange(n, dtype=torch.int32, device=cuda)
                ws = torch.full((vx.lib().vx_sort_workspace_size(n, each),), 0xA5,
                                dtype=torch.uint8, device=cuda)
                vx.sort_pairs(d, v, 32, ws)
                assert vx.workspace_status(ws) == 0
                order = np.argsort(k, kind="stable")
                assert np.array_equal(v.cpu().numpy(), order), (tiles, n)
                assert np.array_equal(d.cpu().numpy().view(dt), k[order]), (tiles, n)
    finally:
        vx.reset_tuning()
