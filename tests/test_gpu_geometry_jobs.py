"""Geometry jobs of two warps: screen-space cache, batch records, clip pool and tile lists against
the oracle at odd job counts, with skinned meshlets and triangles at the near plane, on both sides
of the meshlet count from which a job takes the whole group of eight."""
import numpy as np
import pytest

from compare import compare_frames
from oracle_lib import Oracle
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu

WIDE = 4096     # SFTG_WIDE_JOBS
SUMMED = 2048   # most meshlets whose clip slots need no scan


def _scene(big):
    return scenes.atrium_scene(320, 200, seed=61, nx=15 if big else 5, nz=10 if big else 3, levels=2 if big else 1, arch_segments=16 if big else 8,
                               n_tex=3, tex_size=32, lm_size=1024 if big else 256, n_lights=2, n_chars=3, char_tex=32,
                               floor_quads=(120, 60) if big else (31, 15),
                               views=[(320, 200, (0.2, 0.4, 5.0), (0.5, 2.0, 12.0), np.float32(0.3))])


@pytest.mark.parametrize("big", [False, True])
def test_jobs_equal_oracle(renderer, big):
    sc = _scene(big)
    tss, npx = runtime.scene_counts(sc)
    assert (tss >= WIDE) == big
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, 2)
    finally:
        o.close()
    assert ref["clip"].size > 0
    handle = renderer.load_scene(blob)
    saved = renderer.tuning()
    try:
        renderer.set_samples(2)
        for width in (1, 8) if big else (1, 2, 3, 5, 7, 8):
            renderer.set_tuning(**dict(saved, geom_job_width=width))
            out = renderer.render_debug(handle, 0, tss, npx)
            res = compare_frames(ref, out, 2, len(sc.frames[0].point_lights))
            assert not {k: v for k, v in res.items() if k not in ("color_max_lsb", "tlas") and v != 0}, (width, res)
            if not big:     # batches just under and over the lines
                alone = renderer.render(handle, 0)
                for n in (SUMMED // tss, SUMMED // tss + 1, (WIDE - 1) // tss, (WIDE - 1) // tss + 1):
                    for c in renderer.render_batch([(handle, 0, 2)] * n, [None] * n):
                        assert np.array_equal(c, alone), (width, n)
    finally:
        renderer.set_tuning(**saved)
        renderer.free_scene(handle)
