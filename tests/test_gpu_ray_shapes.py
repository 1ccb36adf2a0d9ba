"""Ray queries where the launch changes shape: one ray, a warp's last ray alone, either side of the
count up to which a ray gets a whole warp; short limits, which drop entries already on the stack;
and a model whose BLAS, given by the caller, has child boxes outside their parent's.  Records equal
the oracle's bit for bit; the caller's tree is compared between the two kernels, ray by ray."""
import ctypes as C

import numpy as np
import pytest

import golden_cases as gc
from oracle_lib import Oracle
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu

WIDE = 81920   # RAY_WIDE_MAX


@pytest.fixture(scope="module")
def atrium(renderer):
    h = renderer.load_scene(gc.blob("atrium_small"))
    yield h
    renderer.free_scene(h)


@pytest.mark.parametrize("n", [1, 3, 31, WIDE, WIDE + 1, WIDE + 18])
def test_ray_counts_match_oracle(renderer, atrium, n):
    r = gc.rays("atrium_small", n=n, seed=500 + n % 97)
    if n > 1:
        r["max_dist"][::3] = np.random.default_rng(n).uniform(0.01, 8.0, len(r["max_dist"][::3]))
    assert renderer.raycast(atrium, r).tobytes() == Oracle(gc.blob("atrium_small")).raycast(r).tobytes()


def test_caller_tree_with_boxes_outside_their_parents(renderer, atrium):
    """The model's own tree with the boxes of every second inner slot shrunk to a quarter: a child's
    box may then be nearer than its parent's, and no stacked entry may be dropped for its own.  The
    narrow kernel (many rays) and the wide one (the same rays in small calls) agree, and differ from
    the answers of the intact tree, so the shrunk boxes matter."""
    sc = gc.scene("atrium_small")
    nodes, root = renderer.model_blas(atrium, 0)
    img = np.frombuffer(nodes, np.uint8).reshape(-1, 256).copy()
    mn, mx = img[:, :96].view(np.float32).reshape(-1, 3, 8), img[:, 96:192].view(np.float32).reshape(-1, 3, 8)
    inner = img[:, 225] == 0
    mid, half = (mn + mx) / 2, (mx - mn) / 8
    shrink = np.zeros(mn.shape, bool)
    shrink[inner, :, ::2] = True
    ok = shrink & (mx >= mn)
    mn[ok], mx[ok] = (mid - half)[ok], (mid + half)[ok]
    keep = []

    class Mesh(C.Structure):
        _fields_ = [("meshlet_count", C.c_uint32), ("attr", C.c_void_p), ("inds", C.c_void_p), ("cull", C.c_void_p), ("joints", C.c_void_p),
                    ("weights", C.c_void_p), ("culling_bones", C.c_void_p), ("material", C.c_int32), ("lightmap_texture", C.c_int32)]

    class Model(C.Structure):
        _fields_ = [("mesh_count", C.c_uint32), ("meshes", C.c_void_p), ("bone_count", C.c_uint32), ("blas_nodes", C.c_void_p),
                    ("blas_count", C.c_uint32), ("blas_root", C.c_uint32), ("build_blas", C.c_uint32)]

    meshes = (Mesh * len(sc.models[0].meshes))()
    for k, ms in enumerate(sc.models[0].meshes):
        arrs = [np.ascontiguousarray(ms.attr, np.float32), np.ascontiguousarray(ms.inds, np.uint8), np.ascontiguousarray(ms.cull, np.float32)]
        keep += arrs
        meshes[k] = Mesh(ms.n, *[a.ctypes.data for a in arrs], None, None, None, -1, -1)
    lib, ctx, out = renderer.lib, renderer.lib.sft_get_gpu_context(), C.c_int32(-1)
    lib.sftg_model_upload.restype, lib.sftg_model_upload.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.c_void_p]
    desc = Model(len(meshes), C.addressof(meshes), 0, img.ctypes.data, len(img), root, 0)
    assert lib.sftg_model_upload(ctx, C.byref(desc), C.byref(out)) == 0
    r = scenes.ray_batch(sc, WIDE + 904, seed=901)
    r["model"] = out.value
    many = renderer.raycast_host(r)
    few = np.concatenate([renderer.raycast_host(r[k:k + 1000]) for k in range(0, len(r), 1000)])
    assert many.tobytes() == few.tobytes()
    r["model"] = renderer.model_device_id(atrium, 0)
    assert renderer.raycast_host(r).tobytes() != many.tobytes()
