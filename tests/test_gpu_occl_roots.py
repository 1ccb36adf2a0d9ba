"""The proxy occlusion pass with a root index outside its tree, TLAS or BLAS: the frame is refused with
the status of a walk that could not be finished, and the next frame is as before."""
import ctypes as C

import numpy as np
import pytest

import caller_trees as ct
import golden_cases as gc
from sofren2_gb300 import runtime
from test_zz_no_alloc import FrameDescHead, lib, _recorded_frame  # noqa: F401

pytestmark = pytest.mark.gpu

SFTG_E_DEVICE_STATUS = -5


class Instance(C.Structure):
    _fields_ = [("model", C.c_int32), ("transform", C.c_float * 16), ("bones", C.c_void_p), ("bone_count", C.c_uint32)]


@pytest.mark.parametrize("tree", ["tlas", "blas"])
@pytest.mark.parametrize("past", [0, 3])
def test_root_outside_its_tree(renderer, lib, tree, past):  # noqa: F811
    h = renderer.load_scene(gc.blob("atrium_small"))
    sc = gc.scene("atrium_small")
    renderer.set_samples(1)
    try:
        want = renderer.render(h, 0)
        nodes, _ = ct.built(renderer, h)
        bad_model = ct.upload(renderer, sc.models[0].meshes, nodes, len(nodes) + past)
        fd = _recorded_frame(renderer, lib, h)
        ctx = lib.sft_get_gpu_context()
        size = 512   # the whole description: the head and the debug texture
        buf = C.create_string_buffer(C.string_at(fd, C.sizeof(FrameDescHead) + 8), size)
        desc = FrameDescHead.from_buffer(buf)
        insts = (Instance * desc.n_instances).from_buffer_copy(C.string_at(desc.instances, C.sizeof(Instance) * desc.n_instances))
        good = renderer.model_device_id(h, 0)
        assert any(i.model == good for i in insts)
        if tree == "tlas":
            desc.tlas_root = desc.tlas_count + past
        else:
            for i in insts:
                if i.model == good:
                    i.model = bad_model
            desc.instances = C.addressof(insts)
        color = np.zeros_like(want)
        assert lib.sftg_frame_render(ctx, C.byref(desc), color.ctypes.data, color.strides[0], None) == SFTG_E_DEVICE_STATUS
        assert lib.sftg_frame_render(ctx, fd, color.ctypes.data, color.strides[0], None) == 0
        assert np.array_equal(color, want)
    finally:
        lib.sft_batch_submit()
        renderer.free_scene(h)
