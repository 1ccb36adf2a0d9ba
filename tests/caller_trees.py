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


class Plates:
    """One meshlet of 120 triangles, one behind the other, each across the z axis."""

    def __init__(self):
        self.n = 1
        attr, inds = np.zeros((10, 64), np.float32), np.zeros((16, 4, 8), np.uint8)
        for q in range(60):
            attr[0:3, q] = ((-9, 9, 0)[q % 3], (-9, -9, 9)[q % 3], 1 + q // 3 / 32)
        for t in range(120):
            p = t % 20
            inds[t >> 3, 0:3, t & 7] = (3 * p, 3 * p + 1, 3 * p + 2) if t // 20 % 2 else (3 * p, 3 * p + 2, 3 * p + 1)
        self.attr, self.inds = attr.reshape(1, -1), inds.reshape(1, -1)
        self.cull = np.array([[0, 0, 1, 20, 0, 0, 1, 2]], np.float32)


def deep_tree(levels, side, slot):
    """A chain of `levels` inner nodes of 8 children, all boxes the same: the chain goes on in `slot`, the other
    children are leaves of 8 triangles or (side "inner") inner nodes of 8 such leaves.  Leaves are shared
    by no two slots."""
    nodes, t = [], [0]

    def add(leaf, kids):
        n = np.zeros(1, NODE)
        n["mn"], n["mx"], n["child"] = 1e30, -1e30, NONE
        n["mn"][:, :, :len(kids)], n["mx"][:, :, :len(kids)] = -9, 9
        n["child"][0, :len(kids)], n["count"], n["leaf"] = kids, len(kids), leaf
        nodes.append(n)
        return len(nodes) - 1

    def leaf():
        t[0] += 1
        return add(1, [TRI | (8 * t[0] + k * 7) % 120 for k in range(8)])

    node = leaf()
    for level in range(levels):
        kids = [leaf() if side == "leaf" else add(0, [leaf() for _ in range(8)]) for _ in range(7)]
        kids.insert(slot, node)
        node = add(0, kids)
    return np.concatenate(nodes), node


def plate_rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros(n, runtime.RAY_DTYPE)
    r["T"] = np.eye(4, dtype=np.float32).reshape(-1)
    r["o"] = np.concatenate([rng.uniform(-2, 2, (n, 2)), rng.uniform(-3, 3, (n, 1))], 1)
    r["d"] = np.concatenate([rng.uniform(-.3, .3, (n, 2)), rng.choice([-1, 1], (n, 1))], 1)
    r["max_dist"] = rng.choice([1.0, 100.0], n)
    return r
