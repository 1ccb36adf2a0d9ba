"""Ray queries against trees that a caller gave: a node index outside the tree marks the record of
every walk that comes to it with hit 2, and both walks (a ray of many, a warp for one of few) give the
same records."""
import numpy as np
import pytest

import caller_trees as ct
import golden_cases as gc
from sofren2_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def atrium(renderer):
    """The scene's handle, its meshes and rays, and an intact copy of its tree behind it in the pool."""
    h = renderer.load_scene(gc.blob("atrium_small"))
    sc = gc.scene("atrium_small")
    yield h, sc.models[0].meshes, scenes.ray_batch(sc, 4000, seed=902)
    renderer.free_scene(h)


@pytest.mark.parametrize("past", [0, 1, 5, ct.TRI - 1, ct.TRI, ct.TRI | 4, ct.NONE - 1, ct.NONE])
def test_root_outside_the_tree(renderer, atrium, past):
    h, meshes, rays = atrium
    nodes, root = ct.built(renderer, h)
    bad = len(nodes) + past if past < 6 else past
    r = rays[:600].copy()
    r["model"] = ct.upload(renderer, meshes, nodes, bad)
    ct.upload(renderer, meshes, nodes, root)
    many, few = ct.cast_both(renderer, r)
    assert (few["hit"] == 2).all() and not ct.differing(many, few)
    assert ct.cast(renderer, r)[0] != 0


@pytest.mark.parametrize("past", [0, 1, 5, ct.TRI - 1, ct.TRI, ct.TRI | 4, ct.NONE - 1])
def test_child_outside_the_tree(renderer, atrium, past):
    """One slot of the root, around everything, with a child that is no node."""
    h, meshes, rays = atrium
    nodes, root = ct.built(renderer, h)
    nodes = nodes[:9].copy()
    nodes[0]["mn"], nodes[0]["mx"], nodes[0]["child"] = -1e4, 1e4, ct.NONE
    nodes[0]["child"][0] = 9 + past if past < 6 else past
    nodes[0]["count"], nodes[0]["leaf"] = 1, 0
    r = rays[:600].copy()
    r["max_dist"] = 1e3
    r["model"] = ct.upload(renderer, meshes, nodes, 0)
    ct.upload(renderer, meshes, ct.built(renderer, h)[0], root)
    many, few = ct.cast_both(renderer, r)
    assert (few["hit"] == 2).all() and not ct.differing(many, few)


@pytest.mark.parametrize("what", ["child", "triangle"])
@pytest.mark.parametrize("every", [2, 3, 7])
def test_walks_that_end_early_beside_others(renderer, atrium, what, every):
    """Rays of an intact tree beside rays, in the same warp, whose walk ends at an index outside the
    model: the former answer as they do alone, the latter are marked."""
    h, meshes, rays = atrium
    nodes, root = ct.built(renderer, h)
    good = rays.copy()
    good["model"] = ct.upload(renderer, meshes, nodes, root)
    want, _ = ct.cast_both(renderer, good)
    one = nodes[:1].copy()
    one["mn"], one["mx"], one["child"] = -1e4, 1e4, ct.NONE
    one["count"], one["leaf"] = 1, what == "triangle"
    one["child"][0, 0] = ct.TRI | sum(m.n for m in meshes) << 7 if what == "triangle" else 1
    r = good.copy()
    r["model"][::every], r["max_dist"][::every] = ct.upload(renderer, meshes, one, 0), 1e3
    for got in ct.cast_both(renderer, r):
        bad = np.arange(len(r)) % every == 0
        assert (got["hit"][bad] == 2).all() and not ct.differing(got[~bad], want[~bad])


@pytest.mark.parametrize("what,one_in", [("child", 40), ("triangle", 4)])
def test_indices_outside_the_model_behind_nearer_hits(renderer, atrium, what, one_in):
    """Some inner children, or leaf triangles, outside the model: the sequential walk skips those that lie
    behind a nearer hit, so some records are answers and some are marked; both walks mark the same."""
    h, meshes, rays = atrium
    nodes, root = ct.built(renderer, h)
    rng = np.random.default_rng(40)
    at = (nodes["leaf"][:, None] == (what == "triangle")) & (np.arange(8) < nodes["count"][:, None]) & (rng.random((len(nodes), 8)) < 1 / one_in)
    at[root] = False
    total = sum(m.n for m in meshes)
    nodes["child"][at] = (ct.TRI | (total + 1) << 7) if what == "triangle" else len(nodes) + 2
    r = rays.copy()
    r["model"] = ct.upload(renderer, meshes, nodes, root)
    many, few = ct.cast_both(renderer, r)
    assert (many["hit"] == 2).sum() > 100 and (many["hit"] == 1).sum() > 100
    assert not ct.differing(many, few)


@pytest.mark.parametrize("levels", [12, 17, 18])
@pytest.mark.parametrize("slot", [7, 3])
def test_deep_trees_whose_boxes_are_all_hit(renderer, levels, slot):
    """Every walk that fits the 128 entries of the walk of many rays fits the one of few."""
    nodes, root = ct.deep_tree(levels, "leaf", slot)
    r = ct.plate_rays(600, levels)
    r["model"] = ct.upload(renderer, [ct.Plates()], nodes, root)
    many, few = ct.cast_both(renderer, r)
    assert not (many["hit"] == 2).any() and (many["hit"] == 1).sum() > 100
    assert not ct.differing(many, few)
