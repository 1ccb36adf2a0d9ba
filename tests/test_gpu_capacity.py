"""A batch that exceeds the payload capacity of a new renderer is rendered again after it has grown: the
views that keep the caller's pixels have to find them as they were, also where the kernels write the
caller's memory in place.  In a process of its own: capacities only grow."""
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
n = 460
sc = scenes.atrium_scene(64, 64, seed=52, nx=16, nz=9, levels=3, arch_segments=8, n_tex=3, tex_size=32, lm_size=512, n_lights=2, n_chars=1,
                         char_tex=32, floor_quads=(60, 30), views=[(64, 64, (0.2, 0.4, 5.0), (0.5, 9.0, 7.0), np.float32(0.3))])
sc.frames[0].clear = 0
with runtime.Renderer(64, 64, 2) as r:
    h = r.load_scene(sc.to_bytes())
    rng = np.random.default_rng(3)
    init = [rng.integers(0, 1 << 32, size=(64, 64), dtype=np.uint32) for _ in range(n)]
    pinned = [torch.zeros((64, 64), dtype=torch.int32).pin_memory() for _ in range(n // 2)]
    bufs = [p.numpy().view(np.uint32) for p in pinned] + [np.zeros((64, 64), np.uint32) for _ in range(n - n // 2)]
    for b, i in zip(bufs, init):
        b[:] = i
    r.render_batch([(h, 0, 2)] * n, bufs)             # over the first capacity: two attempts
    first = [b.copy() for b in bufs]
    out = r.render_debug(h, 0, *runtime.scene_counts(sc))
    assert int(out["tile_payloads"].size) * n > 1 << 20, out["tile_payloads"].size
    assert (first[0] == init[0]).any(), "some of the caller's pixels have to show"
    for k in (0, 1, n // 2 - 1, n // 2, n - 1):
        want = r.render(h, 0, init[k].copy())
        assert np.array_equal(first[k], want), k
print("capacity ok")
'''


def test_kept_pixels_survive_a_second_attempt():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", CODE % (root, os.path.join(root, "tests"))], capture_output=True, text=True, timeout=240)
    assert p.returncode == 0 and "capacity ok" in p.stdout, p.stdout[-2000:] + p.stderr[-2000:]
