"""sftg_frames_render with host buffers and device pointers both asked for: the pointers of views with
pageable buffers, and of views that keep the caller's pixels, are the context's own device memory,
which what the caller does with its buffers afterwards does not reach."""
import ctypes as C
import os

import numpy as np
import pytest

import golden_cases as gc

pytestmark = pytest.mark.gpu


class Attributes(C.Structure):
    _fields_ = [("type", C.c_int), ("device", C.c_int), ("device_pointer", C.c_void_p), ("host_pointer", C.c_void_p), ("reserved", C.c_long * 8)]


@pytest.mark.parametrize("name,pinned", [("small", False), ("variety_noclear", False), ("variety_noclear", True)])
def test_device_pointers_are_device_memory(renderer, name, pinned):
    torch = pytest.importorskip("torch")
    rt = C.CDLL("libcudart.so.13", mode=os.RTLD_NOLOAD | os.RTLD_GLOBAL)
    rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    lib = renderer.lib
    lib.sft_batch_peek.restype, lib.sft_batch_peek.argtypes = C.c_void_p, [C.c_uint32]
    lib.sftg_frames_render.restype, lib.sftg_frames_render.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p]
    h = renderer.load_scene(gc.blob(name))
    renderer.set_samples(1)
    try:
        w, hh = renderer.frame_size(h, 0)
        init = np.random.default_rng(5).integers(0, 1 << 32, size=(hh, w), dtype=np.uint32)
        want = renderer.render(h, 0, init.copy())
        hold = torch.zeros((hh, w), dtype=torch.int32)
        color = (hold.pin_memory() if pinned else hold).numpy().view(np.uint32)
        color[:] = init
        lib.sft_batch_begin()
        assert lib.sftx_scene_render(h, 0, None, 0) == 0
        colors, out = (C.c_void_p * 1)(color.ctypes.data), (C.c_void_p * 1)()
        try:
            assert lib.sftg_frames_render(lib.sft_get_gpu_context(), lib.sft_batch_peek(0), 1, colors, None, out) == 0
            assert np.array_equal(color, want)
            color[:] = 0
            a = Attributes()
            assert rt.cudaPointerGetAttributes(C.byref(a), C.c_void_p(out[0])) == 0 and a.type == 2   # cudaMemoryTypeDevice
            back = np.zeros_like(want)
            assert rt.cudaMemcpy(back.ctypes.data, out[0], back.nbytes, 2) == 0
            assert np.array_equal(back, want)
        finally:
            lib.sft_batch_submit()
    finally:
        renderer.free_scene(h)
