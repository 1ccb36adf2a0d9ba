"""The paths that copy host arrays instead of using them in place, taken here through arrays at odd addresses
(where the GPU shares the host's page tables, nothing else takes them): the same pixels, matrices and
records as in place, at every sample count, with the debug views, and for views that keep the caller's
pixels, alone and beside others over the same buffer in one batch."""
import ctypes as C

import numpy as np
import pytest

import golden_cases as gc
from caller_trees import differing
from oracle_lib import Oracle, lib
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu


def odd(shape, dtype=np.uint32):
    """An array of the type one byte past an aligned address."""
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    a = np.zeros(n + 65, np.uint8)
    start = -a.ctypes.data % 64 + 1
    return a[start:start + n].view(dtype).reshape(shape)


def copied(init):
    a = odd(init.shape, init.dtype)
    a[...] = init
    return a


@pytest.fixture
def scene(renderer):
    live = []

    def load(name):
        live.append(renderer.load_scene(gc.blob(name)))
        w, h = renderer.frame_size(live[-1], 0)
        return live[-1], np.random.default_rng(len(name)).integers(0, 1 << 32, size=(h, w), dtype=np.uint32)

    yield load
    renderer.set_samples(1)
    renderer.set_debug_mode(0)
    for h in live:
        renderer.free_scene(h)


@pytest.mark.parametrize("name", ["small", "config1", "skinned_small", "atrium_small"])
def test_clearing_views(renderer, golden, scene, name):
    h, init = scene(name)
    for S in gc.SAMPLES[name]:
        renderer.set_samples(S)
        got = renderer.render(h, 0, copied(init))
        assert np.array_equal(got, renderer.render(h, 0, init.copy())), S
        assert gc.sha(np.ascontiguousarray(got).reshape(-1)) == golden[name]["samples"][str(S)]["color"], S


@pytest.mark.parametrize("samples", [1, 2, 4])
def test_kept_pixels(renderer, scene, samples):
    """Both paths, and both equal to the oracle over the same pixels."""
    h, init = scene("variety_noclear")
    renderer.set_samples(samples)
    o = Oracle(gc.blob("variety_noclear"))
    try:
        lib().sfto_set_pixels.argtypes = [C.c_void_p, C.c_void_p]
        lib().sfto_set_pixels(o.h, init.ctypes.data)
        want = o.render_color(0, samples, init.shape[1], init.shape[0])[0].reshape(init.shape)
    finally:
        o.close()
    for got in (renderer.render(h, 0, copied(init)), renderer.render(h, 0, init.copy())):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("name", ["variety", "variety_noclear"])
@pytest.mark.parametrize("mode", [1, 2, 3, 4, 5])
def test_debug_views(renderer, scene, name, mode):
    h, init = scene(name)
    renderer.set_debug_mode(mode)
    for S in (1, 2, 4):
        renderer.set_samples(S)
        assert np.array_equal(renderer.render(h, 0, copied(init)), renderer.render(h, 0, init.copy())), S


@pytest.mark.parametrize("samples", [1, 2, 4])
@pytest.mark.parametrize("make", [copied, np.copy])
def test_kept_views_in_one_batch(renderer, scene, samples, make):
    """Each view starts from the pixels before the batch; halves of one picture, and two views over the
    same buffer, which ends as the last one's."""
    h, init = scene("variety_noclear")
    small, _ = scene("small")
    renderer.set_samples(samples)
    hh, w = init.shape
    want = renderer.render(h, 0, init.copy())
    two = make(np.concatenate([init, init], 1))
    renderer.render_batch([(h, 0, samples), (h, 0, samples)], [two[:, :w], two[:, w:]])
    assert np.array_equal(two, np.concatenate([want, want], 1))
    one = make(init)
    renderer.render_batch([(h, 0, 1), (h, 0, 4), (h, 0, samples)], [one, one, one])
    assert np.array_equal(one, want)
    apart = [make(init) for _ in range(3)]
    renderer.render_batch([(h, 0, 1), (h, 0, samples), (h, 0, 4)], apart)
    assert np.array_equal(apart[1], want)
    sw, sh = renderer.frame_size(small, 0)
    room = np.zeros((max(hh, sh), w + sw), np.uint32)
    room[:hh, :w] = init
    room = make(room)
    renderer.render_batch([(h, 0, samples), (small, 0, samples)], [room[:hh, :w], room[:sh, w:]])
    assert np.array_equal(room[:hh, :w], want) and np.array_equal(room[:sh, w:], renderer.render(small, 0))


@pytest.mark.parametrize("lanes", [1, 3])
def test_copied_buffers_on_lanes(renderer, scene, lanes):
    h, init = scene("variety_noclear")
    small, _ = scene("small")
    want, alone = renderer.render(h, 0, init.copy()), renderer.render(small, 0)
    bufs = [copied(init if k % 2 else np.zeros_like(alone)) for k in range(8)]
    renderer.render_batch([((h if k % 2 else small), 0, 1) for k in range(8)], bufs, lanes=lanes)
    for k, b in enumerate(bufs):
        assert np.array_equal(b, want if k % 2 else alone), k


@pytest.mark.parametrize("which", ["requests", "posed", "global", "all"])
@pytest.mark.parametrize("n", [1, 37, 700])
def test_poses(renderer, which, n):
    rig = scenes.pose_rig(6500, n_bones=22)
    sk = renderer.skeleton_upload(rig)
    reqs = scenes.pose_requests(rig, n, seed=n)[:n]          # some name an animation the rig has not
    rec = np.zeros(len(reqs), runtime.POSE_REQUEST_DTYPE)
    rec["skeleton"], rec["animation"], rec["time"] = sk, [a for a, _ in reqs], [t for _, t in reqs]
    out = {"posed": np.full(len(rec) * 22 * 16, 7, np.float32), "global": np.full(len(rec) * 22 * 16, 8, np.float32)}
    got = {k: copied(v) if which in (k, "all") else v.copy() for k, v in out.items()}
    renderer.pose_eval_host(rec, out["posed"], out["global"])
    r = copied(rec) if which in ("requests", "all") else rec
    L = renderer.lib
    assert L.sftg_pose_eval(L.sft_get_gpu_context(), r.ctypes.data, len(r), got["posed"].ctypes.data, got["global"].ctypes.data) == 0
    assert np.array_equal(got["posed"], out["posed"]) and np.array_equal(got["global"], out["global"])


@pytest.mark.parametrize("which", ["rays", "hits", "both"])
@pytest.mark.parametrize("n", [1, 600, 81920])
def test_rays(renderer, scene, which, n):
    h, _ = scene("atrium_small")
    rays = scenes.ray_batch(gc.scene("atrium_small"), n, seed=78)
    rays["model"] = renderer.model_device_id(h, 0)
    want = renderer.raycast_host(rays)
    hits = odd((n,), runtime.HIT_DTYPE) if which != "rays" else np.zeros(n, runtime.HIT_DTYPE)
    r = copied(rays) if which != "hits" else rays
    L = renderer.lib
    assert L.sftg_raycast(L.sft_get_gpu_context(), r.ctypes.data, n, hits.ctypes.data) == 0
    assert not differing(hits.copy(), want)
