"""The raster's parts of a tile's payload list, merged in the visibility buffer, against the oracle:
depth, vis ids and colour of frames whose few tiles hold far more payloads than one part, at every
sample count, with row bands and with the persistent queue; and the tile order of a batch of more
tiles than one CTA orders."""
import numpy as np
import pytest

import golden_cases as gc
from compare import compare_frames
from oracle_lib import Oracle
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples", [1, 2, 4])
@pytest.mark.parametrize("w,h,nx", [(64, 64, 8), (130, 70, 8), (100, 129, 3)])
def test_parts_equal_oracle(renderer, w, h, nx, samples):
    sc = scenes.atrium_scene(w, h, seed=51, nx=nx, nz=4, levels=2, arch_segments=8, n_tex=3, tex_size=32, lm_size=256, n_lights=3, n_chars=1,
                             char_tex=32, floor_quads=(30, 15))
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, samples)
    finally:
        o.close()
    assert int(ref["tile_counts"].max()) > 2 * 64, "a tile's list has to be cut"
    handle = renderer.load_scene(blob)
    saved = renderer.tuning()
    try:
        renderer.set_samples(samples)
        tss, npx = runtime.scene_counts(sc)
        for knobs in ({}, {"tile_queue": 1}, {"raster_bands": (2, 4, 4), "raster_slab_rows": (4, 64, 16)}):
            renderer.set_tuning(**dict(saved, **knobs))
            for _ in range(2):      # a frame after another finds the last one's visibility buffer
                out = renderer.render_debug(handle, 0, tss, npx)
            res = compare_frames(ref, out, samples, len(sc.frames[0].point_lights))
            assert not {k: v for k, v in res.items() if k not in ("color_max_lsb", "tlas") and v != 0}, (knobs, res)
    finally:
        renderer.set_tuning(**saved)
        renderer.free_scene(handle)


@pytest.mark.parametrize("samples", [1, 2, 4])
@pytest.mark.parametrize("w,h", [(60, 30), (150, 200), (960, 832), (1280, 1024)])
def test_bands_of_uncut_lists_equal_oracle(renderer, w, h, samples):
    """1 and 12 tiles (4 bands each), 195 (2), 320 (1) of short lists whose triangles fill them."""
    sc = scenes.atrium_scene(w, h, seed=53, nx=2, nz=1, levels=1, arch_segments=2, n_tex=2, tex_size=16, lm_size=64, n_lights=2, n_chars=0,
                             char_tex=16, floor_quads=(3, 2))
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, samples)
    finally:
        o.close()
    assert 0 < int(np.median(ref["tile_counts"])) < 32
    handle = renderer.load_scene(blob)
    try:
        renderer.set_samples(samples)
        tss, npx = runtime.scene_counts(sc)
        for _ in range(2):
            out = renderer.render_debug(handle, 0, tss, npx)
        res = compare_frames(ref, out, samples, len(sc.frames[0].point_lights))
        assert not {k: v for k, v in res.items() if k not in ("color_max_lsb", "tlas") and v != 0}, res
    finally:
        renderer.free_scene(handle)


def test_order_of_many_tiles(renderer):
    h = renderer.load_scene(gc.blob("small"))
    try:
        w, hh = renderer.frame_size(h, 0)
        tiles = ((w + 63) // 64) * ((hh + 63) // 64)
        n = 8192 // tiles + 2
        alone = {}
        for S in (1, 2, 4):
            renderer.set_samples(S)
            alone[S] = renderer.render(h, 0)
        views = [(h, 0, (1, 2, 4)[k % 3]) for k in range(n)]
        for k, c in enumerate(renderer.render_batch(views, [None] * n)):
            assert np.array_equal(c, alone[views[k][2]]), f"view {k}"
    finally:
        renderer.free_scene(h)


@pytest.mark.parametrize("w,h", [(64, 64), (200, 140), (640, 360)])
def test_binning_segments_equal_oracle(renderer, w, h):
    """Tile lists of a view with more meshlet slots than one segment holds, from one tile (the most
    segments) up, with triangles clipped at the near plane among them."""
    sc = scenes.atrium_scene(w, h, seed=52, nx=16, nz=9, levels=3, arch_segments=8, n_tex=3, tex_size=32, lm_size=512, n_lights=2, n_chars=2,
                             char_tex=32, floor_quads=(60, 30),
                             views=[(w, h, (0.2, 0.4, 5.0), (0.5, 2.0, 12.0), np.float32(0.3))])
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, 1)
    finally:
        o.close()
    tss, npx = runtime.scene_counts(sc)
    assert tss > 1024 and ref["clip"].size > 0
    handle = renderer.load_scene(blob)
    try:
        renderer.set_samples(1)
        out = renderer.render_debug(handle, 0, tss, npx)
        res = compare_frames(ref, out, 1, len(sc.frames[0].point_lights))
        assert not {k: v for k, v in res.items() if k not in ("color_max_lsb", "tlas") and v != 0}, res
        if w == 640:     # in a batch of over 1024 tiles: super-tile lists and no segments
            alone = renderer.render(handle, 0)
            for c in renderer.render_batch([(handle, 0, 1)] * 18, [None] * 18):
                assert np.array_equal(c, alone)
    finally:
        renderer.free_scene(handle)
