"""Host calls whose arrays share bytes: a query's rays and records, a pose call's requests, matrices and
globals.  The results are those of separate arrays (where two outputs share bytes, the globals')."""
import numpy as np
import pytest

import golden_cases as gc
from caller_trees import differing
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def atrium(renderer):
    h = renderer.load_scene(gc.blob("atrium_small"))
    yield h
    renderer.free_scene(h)


@pytest.mark.parametrize("n", [600, 20000])
@pytest.mark.parametrize("at", [0, 1, 64, 100])
def test_records_over_the_rays(renderer, atrium, n, at):
    rays = scenes.ray_batch(gc.scene("atrium_small"), n, seed=77)
    rays["model"] = renderer.model_device_id(atrium, 0)
    want = renderer.raycast_host(rays)
    room = np.zeros(n * 128 + 4096, np.uint8)
    r = room[:n * 96].view(runtime.RAY_DTYPE)
    r[:] = rays
    hits = room[4 * at:4 * at + 32 * n].view(runtime.HIT_DTYPE)
    renderer.raycast_host(r, out=hits)
    assert not differing(hits.copy(), want)


@pytest.fixture(scope="module")
def poses(renderer):
    rig = scenes.pose_rig(6400, n_bones=22)
    sk = renderer.skeleton_upload(rig)
    reqs = [q for q in scenes.pose_requests(rig, 4000, seed=3) if 0 <= q[0] < len(rig["anims"])][:2500]
    rec = np.zeros(len(reqs), runtime.POSE_REQUEST_DTYPE)
    rec["skeleton"], rec["animation"], rec["time"] = sk, [a for a, _ in reqs], [t for _, t in reqs]
    posed, glob = np.zeros((2, len(rec) * 22 * 16), np.float32)
    renderer.pose_eval_host(rec, posed, glob)
    assert (posed != glob).any()
    return rec, posed, glob


def test_globals_over_the_matrices(renderer, poses):
    rec, posed, glob = poses
    both = np.zeros_like(posed)
    renderer.pose_eval_host(rec, both, both)
    assert np.array_equal(both, glob)


@pytest.mark.parametrize("shift", [1, 4, 22 * 16])
def test_globals_over_part_of_the_matrices(renderer, poses, shift):
    rec, posed, glob = poses
    room = np.zeros(len(posed) + shift, np.float32)
    renderer.pose_eval_host(rec, room[:len(posed)], room[shift:])
    assert np.array_equal(room[shift:], glob) and np.array_equal(room[:shift], posed[:shift])


@pytest.mark.parametrize("out", [0, 1])
def test_matrices_over_the_requests(renderer, poses, out):
    rec, posed, glob = poses
    room = [np.zeros_like(posed), np.zeros_like(posed)]
    r = room[out].view(np.uint8)[:rec.nbytes].view(runtime.POSE_REQUEST_DTYPE)
    r[:] = rec
    renderer.pose_eval_host(r, *room)
    assert np.array_equal(room[0], posed) and np.array_equal(room[1], glob)


@pytest.mark.parametrize("out", [0, 1])
def test_matrices_over_requests_some_of_which_leave_them(renderer, poses, out):
    """A request with an animation out of range leaves its matrices, here the bytes of requests, as they were."""
    rec, posed, glob = poses
    bad = rec.copy()
    bad["animation"][::7] = 1000
    room = [np.full_like(posed, 3), np.full_like(posed, 4)]
    r = room[out].view(np.uint8)[:rec.nbytes].view(runtime.POSE_REQUEST_DTYPE)
    r[:] = bad
    before = [x.copy() for x in room]
    renderer.pose_eval_host(r, *room)
    for got, was, want in zip(room, before, (posed, glob)):
        got, was, want = (x.view(np.uint32).reshape(len(rec), -1) for x in (got, was, want))
        left = np.arange(len(rec)) % 7 == 0
        assert np.array_equal(got[left], was[left]) and np.array_equal(got[~left], want[~left])
