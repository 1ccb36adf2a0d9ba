"""Proxy occlusion by static models of every size class of the BLAS walk (walked whole by the first
launch, cut into sub-walks at depth 2, at depth 3), under each other's number of packets, against the
oracle's light_vis: humanoids whose proxies are partly hidden from the lights by spheres."""
import numpy as np
import pytest

from oracle_lib import Oracle
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu


def _scene(slices, bands, lights, chars):
    sc = scenes.skinned_characters_scene(160, 96, seed=71, n_chars=chars, n_lights=lights, tex_size=16, ground_quads=6)
    rng = np.random.default_rng(slices)
    ball = sc.add_model(scenes.Model([scenes.build_meshlets(scenes.uv_sphere(slices, bands, 0.5))], [0]))
    for f in sc.frames:
        for _ in range(10):
            t = scenes.mat_mul(scenes.mat_scale(np.float32(rng.uniform(0.5, 1.6))),
                               scenes.mat_translate(*[np.float32(v) for v in (rng.uniform(-4, 4), rng.uniform(2.2, 4.0), rng.uniform(4, 9))]))
            f.instances.append((ball, t, None))
    return sc, ball


@pytest.mark.parametrize("slices,bands,lights,chars,lo,hi", [(8, 4, 4, 4, 2, 64), (16, 9, 6, 4, 65, 1024), (48, 30, 3, 2, 65, 1024),
                                                             (90, 60, 5, 4, 1025, 1 << 20), (90, 60, 64, 12, 1025, 1 << 20)])
def test_light_vis_equals_oracle(renderer, slices, bands, lights, chars, lo, hi):
    sc, ball = _scene(slices, bands, lights, chars)
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, 1)
        nodes = len(o.model_blas(ball)[0]) // 256
    finally:
        o.close()
    assert lo <= nodes <= hi
    want = ref["light_vis"].reshape(-1, 64)[:, :lights]
    assert len(np.unique(want)) > 1, "some proxies have to be hidden and some not"
    handle = renderer.load_scene(blob)
    try:
        renderer.set_samples(1)
        tss, npx = runtime.scene_counts(sc)
        out = renderer.render_debug(handle, 0, tss, npx)
    finally:
        renderer.free_scene(handle)
    assert np.array_equal(out["light_vis"].reshape(-1, 64)[:, :lights], want)
    assert np.array_equal(out["color"], ref["color"])


@pytest.mark.parametrize("balls", [0, 1, 3, 4, 5, 20, 33, 60])
def test_tlas_sizes_equal_oracle(renderer, balls):
    """TLAS walks of one node up to the 64 instances a frame can hold, four nodes to a step."""
    sc = scenes.skinned_characters_scene(160, 96, seed=72, n_chars=3, n_lights=5, tex_size=16, ground_quads=6)
    rng = np.random.default_rng(balls)
    ball = sc.add_model(scenes.Model([scenes.build_meshlets(scenes.uv_sphere(10, 6, 0.5))], [0]))
    for f in sc.frames:
        for _ in range(balls):
            t = scenes.mat_mul(scenes.mat_scale(np.float32(rng.uniform(0.3, 1.2))),
                               scenes.mat_translate(*[np.float32(v) for v in (rng.uniform(-5, 5), rng.uniform(1.0, 4.5), rng.uniform(3, 10))]))
            f.instances.append((ball, t, None))
        assert len(f.instances) <= 64
    blob = sc.to_bytes()
    o = Oracle(blob)
    try:
        ref = o.render_dump(0, 2)
    finally:
        o.close()
    handle = renderer.load_scene(blob)
    try:
        renderer.set_samples(2)
        tss, npx = runtime.scene_counts(sc)
        out = renderer.render_debug(handle, 0, tss, npx)
    finally:
        renderer.free_scene(handle)
    assert np.array_equal(out["light_vis"].reshape(-1, 64)[:, :5], ref["light_vis"].reshape(-1, 64)[:, :5])
    assert np.array_equal(out["color"], ref["color"])
