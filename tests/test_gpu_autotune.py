"""The autotuner times a knob on work that the knob shapes: the threads per
leaf-parent item on small edits, the longest small list on voxel lists, the
batch's knobs on a batch; and a default stays unless something is faster."""
import pytest

import voxel_b200 as vx
from voxel_b200 import autotune

pytestmark = pytest.mark.gpu


def test_what_is_timed(cuda):
    try:
        res = autotune.main(["--quick", "--quiet", "--out", "/dev/null"])
    finally:
        vx.reset_tuning()
    timed = res["timings_ms"]
    assert not any("lanes" in k for k in timed["edit"])
    blocks, both = vx.tuning_options("edit.leafparent_blocks"), (0, 1)
    for b in blocks:
        for pf in both:
            assert any(f"leafparent_blocks={b} leafparent_prefetch={pf}" in k
                       for k in timed["edit"])
    for knob in ("edit.leafparent_lanes", "edit.small_max_voxels"):
        for v in vx.tuning_options(knob):
            assert any(k.startswith(f"{knob}={v} ") for k in timed["small"])


def test_a_default_stays_unless_beaten():
    assert autotune._pick({1: 1.01, 2: 1.0}, 1) == 1
    assert autotune._pick({1: 1.05, 2: 1.0}, 1) == 2
    assert autotune._pick({1: None, 2: 1.0, 3: 2.0}, 1) == 2
