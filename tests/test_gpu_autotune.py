"""The tuner on views whose size overrules a knob: it leaves there what smaller views are to use, not
whichever of several equal runs was the fastest."""
import numpy as np
import pytest

import golden_cases as gc
from sofren2_gb300 import runtime

pytestmark = pytest.mark.gpu

WIDE = 4096     # SFTG_WIDE_JOBS


@pytest.mark.parametrize("width", [3, 5])
def test_overruled_knobs_stay(renderer, width):
    h = renderer.load_scene(gc.blob("atrium_small"))
    saved = renderer.tuning()
    renderer.set_samples(1)
    try:
        meshlets, _ = runtime.scene_counts(gc.scene("atrium_small"))
        w, hh = renderer.frame_size(h, 0)
        tiles = -(-w // 64) * -(-hh // 64)
        few, many = (WIDE - 1) // meshlets, max(WIDE // meshlets + 1, 1100 // tiles + 1)
        want = renderer.render(h, 0)
        renderer.set_tuning(**dict(saved, geom_job_width=width))
        t = renderer.autotune_batch([(h, 0, 1)] * many, reps=1)
        assert t["geom_job_width"] == width
        assert t["resolve_split"][0] in (16, 2, 1)     # 16, 8 and 4 are the same 4 CTAs from 1024 tiles on
        assert np.array_equal(renderer.render(h, 0), want)
        t = renderer.autotune_batch([(h, 0, 1)] * few, reps=1)
        assert t["geom_job_width"] in (1, 2, 4, 8)
    finally:
        renderer.set_tuning(**saved)
        renderer.free_scene(h)
