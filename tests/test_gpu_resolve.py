"""The resolve's fragment lists against the oracle, pixel for pixel: triangles smaller than a pixel
(many fragments of many triangles in one 4x2 block), frame edges inside a block, every number of
CTAs per tile, and lights and proxies whose products with zero are not zero (infinite colour, zero
radius), where uncovered pixels of a block decide with the covered ones."""
import numpy as np
import pytest

from oracle_lib import Oracle
from sofren2_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(kind, w, h):
    if kind == "atrium":
        sc = scenes.atrium_scene(w, h, seed=41, nx=6, nz=4, levels=2, arch_segments=6, n_tex=4, tex_size=64, lm_size=128, n_lights=9,
                                 n_chars=2, char_tex=64, floor_quads=(24, 12))
    else:
        sc = scenes.skinned_characters_scene(w, h, seed=42, n_chars=4, n_lights=6, tex_size=64, ground_quads=40)
    if kind != "odd":
        return sc
    for f in sc.frames:    # an infinite colour of short reach, a light without reach, a dim one far out
        (p0, *_), (p1, *_) = f.point_lights[0], f.point_lights[1]
        near = (p0[0], np.float32(1.2), p0[2])
        f.point_lights[0] = (near, np.float32(3e38), np.float32(3e38), np.float32(0.5), np.float32(10.0), np.float32(2.5))
        f.point_lights[1] = (p1, np.float32(0.5), np.float32(0.5), np.float32(0.5), np.float32(1.0), np.float32(0.0))
    for m in sc.models:    # proxies of zero size among the others
        m.proxies = [(a, a if k % 3 == 0 else b, 0.0 if k % 3 == 0 else r, bone) for k, (a, b, r, bone) in enumerate(m.proxies)]
    return sc


@pytest.mark.parametrize("samples", [1, 2, 4])
@pytest.mark.parametrize("kind,w,h", [("skinned", 65, 67), ("skinned", 150, 34), ("atrium", 129, 71), ("odd", 131, 66)])
def test_resolve_equals_oracle(renderer, kind, w, h, samples):
    sc = _scene(kind, w, h)
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        want = np.asarray(o.render_dump(0, samples)["color"]).reshape(h, w)
    finally:
        o.close()
    handle = renderer.load_scene(blob)
    saved = renderer.tuning()
    try:
        renderer.set_samples(samples)
        for split, lists in ((16, 0), (8, 1), (4, 2), (1, 1)):
            renderer.set_tuning(**dict(saved, resolve_split=(split,) * 3, tile_lights=(lists,) * 3))
            got = renderer.render(handle, 0)
            assert np.array_equal(got, want), f"{int(np.count_nonzero(got != want))} pixels differ with {split} CTAs per tile"
    finally:
        renderer.set_tuning(**saved)
        renderer.free_scene(handle)
