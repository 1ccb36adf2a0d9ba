"""Batches on submission lanes and the colour buffers they share: one with a view that keeps the caller's
pixels has completed when its submission returns, so that batches composed over one buffer, on any
lanes, are drawn in the order they were submitted."""
import numpy as np
import pytest

import golden_cases as gc

pytestmark = pytest.mark.gpu


def _submit(r, lane, views):
    """views: (scene handle, frame, colour array)."""
    r.lib.sft_batch_begin()
    for h, f, c in views:
        assert r.lib.sftx_scene_render(h, f, c.ctypes.data, c.strides[0]) == 0
    assert r.lib.sft_batch_submit_async(lane) == 0


@pytest.fixture(scope="module")
def kept(renderer):
    h = renderer.load_scene(gc.blob("variety_noclear"))
    w, hh = renderer.frame_size(h, 0)
    init = np.random.default_rng(9).integers(0, 1 << 32, size=(hh, w), dtype=np.uint32)
    yield h, init
    renderer.free_scene(h)


def _buffers(shape, pinned, n):
    torch = pytest.importorskip("torch")
    if not pinned:
        return None, [np.zeros(shape, np.uint32) for _ in range(n)]
    keep = [torch.zeros(shape, dtype=torch.int32).pin_memory() for _ in range(n)]
    return keep, [t.numpy().view(np.uint32) for t in keep]


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("samples", [1, 4])
def test_kept_pixels_are_drawn_when_the_submission_returns(renderer, kept, pinned, samples):
    h, init = kept
    renderer.set_samples(samples)
    try:
        want = renderer.render(h, 0, init.copy())
        hold, bufs = _buffers(init.shape, pinned, 60)
        for b in bufs:
            b[:] = init
        _submit(renderer, 1, [(h, 0, b) for b in bufs])
        last = bufs[-1].copy()
        assert renderer.lib.sft_batch_done(1) == 1 and np.array_equal(last, want)
        assert renderer.lib.sft_batch_wait(1) == 0
        assert all(np.array_equal(b, want) for b in bufs)
    finally:
        renderer.set_samples(1)


@pytest.mark.parametrize("pinned", [False, True])
def test_kept_batches_over_one_buffer_follow_one_another(renderer, kept, pinned):
    """Blending is not idempotent at 4x: four batches on four lanes over the same buffers equal four lone
    renders."""
    h, init = kept
    renderer.set_samples(4)
    try:
        want = init.copy()
        steps = [want.copy()]
        for _ in range(4):
            steps.append(renderer.render(h, 0, want).copy())
        assert (steps[-1] != steps[-2]).any()
        hold, bufs = _buffers(init.shape, pinned, 20)
        for b in bufs:
            b[:] = init
        for lane in (1, 2, 3, 4):
            _submit(renderer, lane, [(h, 0, b) for b in bufs])
        for lane in (1, 2, 3, 4):
            assert renderer.lib.sft_batch_wait(lane) == 0
        assert all(np.array_equal(b, steps[-1]) for b in bufs)
    finally:
        renderer.set_samples(1)


@pytest.mark.parametrize("where", ["same", "rows", "corner"])
@pytest.mark.parametrize("second", ["lane", "call", "kept"])
def test_later_batches_over_pageable_buffers_win(renderer, kept, where, second):
    """A long batch on one lane, whose last view goes to a buffer that the next submission, or a call on the
    synchronous lane, draws over: the buffer ends as if the two had run one after the other."""
    keep_h, init = kept
    big, small = renderer.load_scene(gc.blob("atrium_small")), renderer.load_scene(gc.blob("small"))
    try:
        renderer.set_samples(1)
        w, h = renderer.frame_size(big, 0)
        over = keep_h if second == "kept" else small
        w2, h2 = renderer.frame_size(over, 0)
        room = np.zeros((h + h2 + 4, w + w2 + 4), np.uint32)
        a, at = room[2:2 + h, 2:2 + w], {"same": (2, 2), "rows": (2 + h // 2, 2), "corner": (1 + h, 1 + w)}[where]
        b = room[at[0]:at[0] + h2, at[1]:at[1] + w2]
        renderer.render(big, 0, a)
        renderer.render(over, 0, b)
        want = room.copy()
        assert (want[2:2 + h, 2:2 + w] != 0).any()
        for _ in range(3):
            room[:] = 0
            others = [np.zeros((h, w), np.uint32) for _ in range(60)]
            _submit(renderer, 1, [(big, 0, c) for c in others] + [(big, 0, a)])
            if second == "call":
                renderer.render(over, 0, b)
            else:
                _submit(renderer, 2, [(over, 0, b)])
                assert renderer.lib.sft_batch_wait(2) == 0
            assert renderer.lib.sft_batch_wait(1) == 0
            assert np.array_equal(room, want)
    finally:
        renderer.free_scene(big)
        renderer.free_scene(small)
