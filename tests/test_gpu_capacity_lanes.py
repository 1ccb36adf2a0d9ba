"""Two batches submitted before either is waited for (one that keeps the caller's pixels has completed by
then), both over the first payload capacity of a new renderer: the first one waited for grows the
capacities, and the second has to be rendered again all the same.  In a process of its own: capacities
only grow."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = r'''
import sys
sys.path[:0] = [r"%s", r"%s"]
import numpy as np, torch
from sofren2_gb300 import runtime, scenes
n, first, clear = 460, int(sys.argv[1]), int(sys.argv[2])
def scene(clear):
    sc = scenes.atrium_scene(64, 64, seed=52, nx=16, nz=9, levels=3, arch_segments=8, n_tex=3, tex_size=32, lm_size=512, n_lights=2, n_chars=1,
                             char_tex=32, floor_quads=(60, 30), views=[(64, 64, (0.2, 0.4, 5.0), (0.5, 9.0, 7.0), np.float32(0.3))])
    sc.frames[0].clear = clear
    return sc
with runtime.Renderer(64, 64, 2) as r:
    hs = [r.load_scene(scene(c).to_bytes()) for c in (clear, 1)]     # lanes 1 and 2
    rng = np.random.default_rng(4)
    init = rng.integers(0, 1 << 32, size=(64, 64), dtype=np.uint32)
    keep = [[torch.zeros((64, 64), dtype=torch.int32).pin_memory() for _ in range(n // 2)] for _ in hs]
    bufs = [[p.numpy().view(np.uint32) for p in k] + [np.zeros((64, 64), np.uint32) for _ in range(n - n // 2)] for k in keep]
    for b in bufs[0] + bufs[1]:
        b[:] = init
    for lane in (1, 2):
        r.lib.sft_batch_begin()
        for b in bufs[lane - 1]:
            assert r.lib.sftx_scene_render(hs[lane - 1], 0, b.ctypes.data, b.strides[0]) == 0
        assert r.lib.sft_batch_submit_async(lane) == 0
    for lane in (first, 3 - first):
        assert r.lib.sft_batch_wait(lane) == 0
    out = r.render_debug(hs[1], 0, *runtime.scene_counts(scene(1)))
    assert int(out["tile_payloads"].size) * n > 1 << 20, out["tile_payloads"].size
    for h, bs in zip(hs, bufs):
        want = r.render(h, 0, init.copy())
        assert (want != init).any()
        wrong = [k for k, b in enumerate(bs) if not np.array_equal(b, want)]
        assert not wrong, (bs is bufs[0], wrong[:5], len(wrong))
print("lanes ok")
'''


@pytest.mark.parametrize("first", [1, 2])
@pytest.mark.parametrize("clear", [0, 1])
def test_both_lanes_over_capacity(first, clear):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", CODE % (root, os.path.join(root, "tests")), str(first), str(clear)], capture_output=True, text=True, timeout=240)
    assert p.returncode == 0 and "lanes ok" in p.stdout, p.stdout[-2000:] + p.stderr[-2000:]
