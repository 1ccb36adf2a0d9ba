"""Models with a BLAS given by the caller (sftg_model_upload's blas_nodes), for the GPU tests."""
import ctypes as C

import numpy as np

from sofren2_gb300 import runtime

NODE = np.dtype([("mn", "<f4", (3, 8)), ("mx", "<f4", (3, 8)), ("child", "<u4", (8,)), ("count", "u1"), ("leaf", "u1"), ("pad", "u1", (30,))])
NONE, TRI = 0xFFFFFFFF, 0x80000000
WIDE = 81920   # SFTG_RAY_WIDE_MAX


class Mesh(C.Structure):
    _fields_ = [("meshlet_count", C.c_uint32), ("attr", C.c_void_p), ("inds", C.c_void_p), ("cull", C.c_void_p), ("joints", C.c_void_p),
                ("weights", C.c_void_p), ("culling_bones", C.c_void_p), ("material", C.c_int32), ("lightmap_texture", C.c_int32)]


class Model(C.Structure):
    _fields_ = [("mesh_count", C.c_uint32), ("meshes", C.c_void_p), ("bone_count", C.c_uint32), ("blas_nodes", C.c_void_p),
                ("blas_count", C.c_uint32), ("blas_root", C.c_uint32), ("build_blas", C.c_uint32)]


def upload(renderer, meshes, nodes, root=0):
    """The resident id of a model of scenes meshes with the node images `nodes` (NODE records)."""
    keep, ms = [nodes], (Mesh * len(meshes))()
    for k, m in enumerate(meshes):
        arrs = [np.ascontiguousarray(m.attr, np.float32), np.ascontiguousarray(m.inds, np.uint8), np.ascontiguousarray(m.cull, np.float32)]
        keep += arrs
        ms[k] = Mesh(m.n, *[a.ctypes.data for a in arrs], None, None, None, -1, -1)
    lib, out = renderer.lib, C.c_int32(-1)
    lib.sftg_model_upload.restype, lib.sftg_model_upload.argtypes = C.c_int, [C.c_void_p, C.c_void_p, C.c_void_p]
    desc = Model(len(meshes), C.addressof(ms), 0, nodes.ctypes.data, len(nodes), root, 0)
    assert lib.sftg_model_upload(lib.sft_get_gpu_context(), C.byref(desc), C.byref(out)) == 0
    return out.value


def built(renderer, handle, mi=0):
    """(node records, root) of a scene's model as built here."""
    img, root = renderer.model_blas(handle, mi)
    return np.frombuffer(img, NODE).copy(), root


def cast(renderer, rays):
    """(status, records) of sftg_raycast; a status of 0 has no overflowed walk."""
    out = np.zeros(len(rays), runtime.HIT_DTYPE)
    r = np.ascontiguousarray(rays, runtime.RAY_DTYPE)
    return renderer.lib.sftg_raycast(renderer.lib.sft_get_gpu_context(), r.ctypes.data, len(r), out.ctypes.data), out


def cast_both(renderer, rays):
    """The records by the walk of many rays (rays repeated past the line) and by that of few."""
    times = WIDE // len(rays) + 1
    many = cast(renderer, np.tile(rays, times))[1][:len(rays)]
    few = np.concatenate([cast(renderer, rays[k:k + 1000])[1] for k in range(0, len(rays), 1000)])
    return many, few


def differing(a, b):
    """Indices of the records that differ in any bit."""
    return np.flatnonzero((a.view(np.uint8).reshape(len(a), -1) != b.view(np.uint8).reshape(len(b), -1)).any(1)).tolist()
