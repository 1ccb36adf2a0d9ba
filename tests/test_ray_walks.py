"""The two ray walks (sofren2_gb300/csrc/sftg_ray.cu) on the CPU, lane by lane (warp_sim.h), on trees a
caller may give: they end, their lanes meet at every collective, nothing outside the tree is read, and the
records of both are the same."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import golden_cases as gc
from caller_trees import NODE, NONE, TRI, Plates, deep_tree, differing, plate_rays
from oracle_lib import Oracle
from sofren2_gb300 import runtime, scenes

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "sofren2_gb300", "csrc")


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    tmp = tmp_path_factory.mktemp("walks")
    ray, blas = (open(os.path.join(CSRC, f)).read() for f in ("sftg_ray.cu", "sftg_blas.cu"))
    (tmp / "ray_body.inc").write_text(ray[ray.index("#define RAY_STACK"):ray.index("#define RAY_GRID")])
    (tmp / "forms_body.inc").write_text(blas[blas.index("__global__ void k_blas_walk_forms"):blas.index("void sftg_launch_walk_forms")])
    exe = str(tmp / "ray_walks")
    subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-ffp-contract=off", "-Wno-unused-function", "-fsanitize=address", "-I", str(tmp), "-I", HERE,
                    "-I", CSRC, "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "ray_walks.cc"), "-o", exe], check=True)
    return exe


def run(exe, tmp_path, nodes, root, meshes, rays, nested):   # nested 2: as an upload finds
    path, out = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    with open(path, "wb") as f:
        np.array([len(nodes), root, sum(m.n for m in meshes), len(rays), nested], np.uint32).tofile(f)
        nodes.tofile(f)
        for m in meshes:
            np.ascontiguousarray(m.attr, np.float32).tofile(f)
        for m in meshes:
            np.ascontiguousarray(m.inds, np.uint8).tofile(f)
        rays.tofile(f)
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:detect_stack_use_after_return=0")
    p = subprocess.run([exe, path, out], capture_output=True, text=True, timeout=300, env=env)
    assert p.returncode == 0, p.stdout[-500:] + p.stderr[-1500:]
    rec = np.fromfile(out, runtime.HIT_DTYPE)
    return rec[:len(rays)], rec[len(rays):]


@pytest.fixture(scope="module")
def atrium():
    sc = gc.scene("atrium_small")
    o = Oracle(gc.blob("atrium_small"))
    try:
        img, root = o.model_blas(0)
        rays = scenes.ray_batch(sc, 200, seed=903)
        rays["model"] = 0
        want = o.raycast(rays)
    finally:
        o.close()
    return np.frombuffer(img, NODE).copy(), root, sc.models[0].meshes, rays, want


def test_sound_tree_matches_oracle(walks, atrium, tmp_path):
    nodes, root, meshes, rays, want = atrium
    assert (want["hit"] == 1).sum() > 20
    for nested in (0, 1, 2):
        for got in run(walks, tmp_path, nodes, root, meshes, rays, nested):
            assert not differing(got, want)


@pytest.mark.parametrize("what,bad", [("triangle", 0), ("triangle", NONE - 1), ("child", 0), ("child", TRI), ("child", TRI | 5), ("child", NONE - 1)])
def test_indices_outside_the_model(walks, atrium, tmp_path, what, bad):
    """One in 20 inner children, or one in 4 triangles, outside the model, so that walks end early beside others of their warp."""
    nodes, root, meshes, rays, _ = atrium
    n = nodes.copy()
    at = (n["leaf"][:, None] == (what == "triangle")) & (np.arange(8) < n["count"][:, None])
    at &= np.random.default_rng(20).random(at.shape) < (1 / 4 if what == "triangle" else 1 / 20)
    at[root] = False
    n["child"][at] = bad or (TRI | sum(m.n for m in meshes) << 7 if what == "triangle" else len(n))
    many, few = run(walks, tmp_path, n, root, meshes, rays, 2)
    assert (many["hit"] == 2).sum() > 3 and (many["hit"] == 1).sum() > 10
    assert not differing(many, few)


@pytest.mark.parametrize("root", [0, 1, TRI - 1, TRI, TRI | 9, NONE])
def test_root_outside_the_tree(walks, atrium, tmp_path, root):
    nodes, _, meshes, rays, _ = atrium
    many, few = run(walks, tmp_path, nodes, len(nodes) + root if root < 2 else root, meshes, rays[:40], 0)
    assert (many["hit"] == 2).all() and not differing(many, few)


@pytest.mark.parametrize("levels", [1, 12, 16, 17, 18])
@pytest.mark.parametrize("side,slot", [("leaf", 7), ("leaf", 3), ("inner", 7)])
def test_deep_trees_whose_boxes_are_all_hit(walks, tmp_path, levels, side, slot):
    """Every walk that fits the 128 entries of the walk of many rays fits the one of few."""
    levels -= side == "inner" and levels == 18     # a level more of its own
    nodes, root = deep_tree(levels, side, slot)
    many, few = run(walks, tmp_path, nodes, root, [Plates()], plate_rays(8, levels), 2)
    assert not (many["hit"] == 2).any() and (many["hit"] == 1).any()
    assert not differing(many, few)
