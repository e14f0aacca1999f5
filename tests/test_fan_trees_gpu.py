"""The fan layout (sr_fan.cuh) on what an upload may hold. It leaves boxes of the tree out, which a ray does not
notice where boxes are nested: where they are not, frames and caller rays must still be the reference's walk over
every box. Records may hold NaNs and infinities, which pass the ray test's comparisons."""
import numpy as np
import pytest

import specrel_b200 as sr

pytestmark = pytest.mark.gpu

IDX = 43
UP = 2.0 ** 41  # a power of two: hits of the scaled ray are the ray's, divided; past the layouts' range of values


def _tree(shrink):
    """The 147,456-tetrahedron cube scene (too large for the lone walk) with one inner box in seven of levels 3 to 9
    shrunk to a part of itself."""
    p = sr.synth_scene(1, 5, n_bodies=64).packed()
    nodes = p.nodes.copy()
    depth = np.zeros(len(nodes), int)
    for i in range(len(nodes)):
        if nodes["count"][i] == 0:
            depth[nodes["left"][i]] = depth[nodes["right_or_first"][i]] = depth[i] + 1
    pick = np.flatnonzero((nodes["count"] == 0) & (depth >= 3) & (depth <= 9))[::7]
    if shrink:
        lo, hi = nodes["min"][pick], nodes["max"][pick]
        nodes["min"][pick], nodes["max"][pick] = lo + 0.3 * (hi - lo), hi - 0.3 * (hi - lo)
    return sr.PackedScene(nodes, p.geoms, p.attrs, p.materials, p.stars, 0, p.light_pos, p.leaf_to_orig)


def _same(a, b):
    assert (a.hit_id == b.hit_id).all() and (a.lam.view(np.uint32) == b.lam.view(np.uint32)).all() and (a.rgb == b.rgb).all()


@pytest.mark.parametrize("shrink", [False, True])
def test_boxes_that_do_not_hold_their_childrens(engine, shrink):
    packed = _tree(shrink)
    engine.upload(IDX, packed)
    hits = 0
    for pos in ((0.0, 0.0, 0.0, 0.0), (-20.0, 5.0, 3.0, -4.0), (-40.0, -10.0, 6.0, 2.0)):
        for shadow in (0, 1):
            u = sr.uniforms(sr.camera(pos, 110.0, rapidity=(0.4, 0.1, -0.3)), 640, 400, 0, shadow, 0,
                            num_nodes=len(packed.nodes), light_pos=packed.light_pos)
            fast, plain = (engine.render(IDX, u, path=path, aux=True) for path in (sr.SR_PATH_FAST, sr.SR_PATH_PLAIN))
            _same(fast, plain)
            hits += int((plain.hit_id != 0xFFFFFFFF).sum())
    assert hits > 0


@pytest.mark.parametrize("shrink", [False, True])
def test_caller_rays_into_such_a_tree(engine, shrink):
    engine.upload(IDX, _tree(shrink))
    rng = np.random.default_rng(4)
    d = rng.normal(size=(3000, 3))
    rays = np.zeros((3000, 10))
    rays[:, 4], rays[:, 5:8] = -1.0, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays = rays.astype(np.float32).astype(np.float64)
    rays[:, 8], rays[:, 9] = np.float32(1e-3), 180.0
    far = rays.copy()
    far[:, 4:8] *= UP
    far[:, 8:10] /= UP
    a, b = engine.trace_rays(IDX, rays), engine.trace_rays(IDX, far)
    assert (a["slot"] == b["slot"]).all() and (a["lambda_"] == b["lambda_"] * np.float32(UP)).all()
    assert (a["slot"] != 0xFFFFFFFF).any()


def _broken(row, value):
    """Every seventh record with a row of its barycentric matrix set to `value`; hit ids are leaf slots."""
    p = _tree(False)
    geoms = p.geoms.copy()
    geoms.view(np.float32).reshape(-1, 5, 4)[::7, row] = value
    return sr.PackedScene(p.nodes, geoms, p.attrs, p.materials, p.stars, 0, p.light_pos, None)


def _early(packed, u, pixels, slots, lam):
    """Whether a hit lies before the entry of its leaf's box, where the packet's order need not be the reference's
    (SrTuning.packet's condition); by the ray and the box in 64 bits, up to a rounding of 1e-5."""
    leaf = np.flatnonzero(packed.nodes["count"] > 0)
    leaf = leaf[np.argsort(packed.nodes["right_or_first"][leaf])]
    first = packed.nodes["right_or_first"][leaf]
    w, h = u.size[0], u.size[1]
    e = np.array([list(r) for r in u.e])
    out = np.zeros(len(pixels), bool)
    for k, (pix, slot, la) in enumerate(zip(pixels, slots, lam)):
        if slot == 0xFFFFFFFF:
            continue
        n = np.array([(2.0 * (pix % w + 0.5) / w - 1.0) * u.half_wh[0], (1.0 - 2.0 * (pix // w + 0.5) / h) * u.half_wh[1], 1.0])
        n /= np.linalg.norm(n)
        d = -e[0] + n[0] * e[1] + n[1] * e[2] + n[2] * e[3]
        node = packed.nodes[leaf[np.searchsorted(first, slot, "right") - 1]]
        a, b = (node["min"] - np.array(list(u.cam_pos))) / d, (node["max"] - np.array(list(u.cam_pos))) / d
        out[k] = la < np.minimum(a, b).max() * (1.0 + 1e-5)
    return out


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("row", [2, 3, 4])
def test_records_with_nans_and_infinities(engine, row, value):
    """Such a record is hit over more of its hyperplane than its tetrahedron. Pixels may differ from the reference's
    only where one of the two hits lies before its leaf's box is entered."""
    packed = _broken(row, value)
    engine.upload(IDX, packed)
    hits = broken = 0
    for pos in ((0.0, 0.0, 0.0, 0.0), (-20.0, 5.0, 3.0, -4.0)):
        u = sr.uniforms(sr.camera(pos, 110.0, rapidity=(0.4, 0.1, -0.3)), 640, 400, 0, 0, 0,
                        num_nodes=len(packed.nodes), light_pos=packed.light_pos)
        fast, plain = (engine.render(IDX, u, path=path, aux=True) for path in (sr.SR_PATH_FAST, sr.SR_PATH_PLAIN))
        diff = np.flatnonzero(fast.hit_id != plain.hit_id)
        early = _early(packed, u, diff, fast.hit_id[diff], fast.lam[diff]) | _early(packed, u, diff, plain.hit_id[diff], plain.lam[diff])
        assert early.all()
        hit = plain.hit_id != 0xFFFFFFFF
        hits += int(hit.sum())
        broken += int((hit & (plain.hit_id % 7 == 0)).sum())
    assert broken > hits / 10  # they are met often


@pytest.mark.parametrize("steps", ["frame", "rays", "lone frame", "lone rays frame", "layout frame", "rays layout rays frame",
                                   "update lone frame rays", "rays update update rays frame"])
def test_small_scenes_get_the_layout_when_wanted(engine, steps):
    """A scene of at most 2^17 records has its fan layout made by the first large frame or list of rays after each
    change: every order of changes and uses gives the plain path's frames and the same rays' hits."""
    s = sr.synth_scene(1, 1, n_bodies=16)
    p = s.packed()
    engine.build_tubes(IDX, s)
    rays = np.zeros((20000, 10))
    d = np.random.default_rng(7).normal(size=(20000, 3))
    rays[:, 0:4], rays[:, 4], rays[:, 5:8] = (-20.0, 5.0, 3.0, -4.0), -1.0, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 8], rays[:, 9] = 1e-3, 180.0
    far = rays.copy()
    far[:, 4:8], far[:, 8:10] = rays[:, 4:8].astype(np.float32) * np.float64(UP), rays[:, 8:10].astype(np.float32) / np.float64(UP)
    for layout, step in enumerate(steps.split()):
        if step == "update":
            engine.update(IDX, s, node_ranges=[(0, len(p.nodes))], prim_ranges=[(0, len(p.geoms))])
        elif step == "layout":
            engine.set_layout(IDX, 1 + layout % 2)
        elif step == "rays":
            a, b = engine.trace_rays(IDX, rays), engine.trace_rays(IDX, far)
            assert (a["slot"] == b["slot"]).all() and (a["slot"] != 0xFFFFFFFF).any()
        else:
            w, h = (1920, 1200) if step == "frame" else (320, 200)
            u = sr.uniforms(sr.camera((-20.0, 5.0, 3.0, -4.0), 100.0, rapidity=(0.4, 0.1, -0.3)), w, h, 0, 1, 0,
                            num_nodes=s.num_nodes, light_pos=s.light_pos)
            fast, plain = (engine.render(IDX, u, path=path, aux=True) for path in (sr.SR_PATH_FAST, sr.SR_PATH_PLAIN))
            _same(fast, plain)
            assert (plain.hit_id != 0xFFFFFFFF).any()
    engine.set_layout(IDX, 0)
