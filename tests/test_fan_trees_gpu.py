"""The fan layout (sr_fan.cuh) leaves boxes of the tree out, which a ray does not notice where boxes are nested. An
uploaded tree need not be: its frames and caller rays must still be the reference's walk over every box."""
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
