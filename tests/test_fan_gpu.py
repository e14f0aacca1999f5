"""The packet walk over the fan layout (sr_fan.cuh) where it can go wrong: every tile shape, frames that
are not a multiple of a tile, views whose rays spread so far that tiles are given up and walked in
groups, shadow walks that are given up and finished ray by ray, leaves of up to 63 records.
Every frame's hit records, lambda, tau and RGB must equal the per-ray walk's bit for bit
(exact by construction: the packet tests the same records with the same arithmetic)."""
import ctypes as C

import numpy as np
import pytest

import specrel_b200 as sr
from specrel_b200 import _lib as L

pytestmark = pytest.mark.gpu

IDX, BIG = 41, 42


@pytest.fixture(scope="module")
def bodies(engine):
    s = sr.synth_scene(2, 3, n_bodies=8)
    engine.build_tubes(IDX, s)
    return s


def _both(engine, idx, u, cam, **tile):
    keep = engine.tuning(idx)
    out = []
    try:
        for packet in (0, 1):
            t = engine.tuning(idx)
            t.packet = packet
            for k, v in tile.items():
                setattr(t, k, v)
            engine.set_tuning(idx, t)
            out.append(engine.render(idx, u, aux=True, cam=cam))
    finally:
        engine.set_tuning(idx, keep)
    a, b = out
    for x, y in ((a.hit_id, b.hit_id), (a.lam.view(np.uint32), b.lam.view(np.uint32)),
                 (a.tau.view(np.uint32), b.tau.view(np.uint32)), (a.rgb, b.rgb)):
        assert (x == y).all()
    return b


def _u(scene, w, h, rapidity=(0.0, 0.0, 0.0), pos=(0.0, 0.0, 0.0, 0.0), fov=90.0, slice_mode=0, shadow=1):
    cam = sr.camera(pos, fov, rapidity=rapidity)
    u = sr.uniforms(cam, w, h, 0, shadow, slice_mode, num_nodes=scene.num_nodes, light_pos=scene.light_pos)
    return u, sr.cam64(pos, rapidity)


@pytest.mark.parametrize("tile", [(1, 32), (2, 16), (4, 8), (8, 4), (16, 2), (32, 1)])
def test_tile_shapes_and_ragged_frames(engine, bodies, tile):
    for w, h in ((1, 1), (9, 7), (65, 33), (161, 95)):
        u, cam = _u(bodies, w, h, (0.3, -0.2, 0.4))
        _both(engine, IDX, u, cam, tile_w=tile[0], tile_h=tile[1])


@pytest.mark.parametrize("slice_mode", [0, 1, 2, 3])
@pytest.mark.parametrize("rapidity", [(0.0, 0.0, 0.0), (1.6, -1.4, 1.2), (-2.0, 1.0, -2.0)])
def test_spread_rays_are_split(engine, bodies, slice_mode, rapidity):
    """Small frames with a wide field of view seen by fast observers: tiles span whole bodies."""
    hits = 0
    for fov in (60.0, 150.0):
        u, cam = _u(bodies, 95, 41, rapidity, fov=fov, slice_mode=slice_mode, shadow=2 if slice_mode == 1 else 1)
        hits += int((_both(engine, IDX, u, cam).hit_id != 0xFFFFFFFF).sum())
    print("hits", hits)


@pytest.mark.parametrize("shadow", [1, 2])
def test_shadow_rays(engine, bodies, shadow):
    for seed in range(4):
        rng = np.random.default_rng(seed)
        u, cam = _u(bodies, 201, 131, tuple(rng.uniform(-1.0, 1.0, 3)), pos=(0.0,) + tuple(rng.uniform(-2.0, 2.0, 3)), shadow=shadow)
        _both(engine, IDX, u, cam)


@pytest.mark.parametrize("group", [1, 5, 11, 16, 21])  # largest leaves: 6, 15, 33, 48, 63
def test_large_leaves(engine, bodies, group):
    """The same records under trees over groups of `group` of them, so that leaves hold up to 63: more than a
    warp has lanes, and all a node reference can name."""
    boxes, geoms, attrs, p = sr.synth_scene(1, 5, n_bodies=64).build_inputs()  # too large for small frames' own walk
    assert len(geoms) > 1 << 17
    n = len(geoms)
    starts = np.arange(0, n, group)
    lo = np.minimum.reduceat(boxes[:, :4], starts, axis=0)
    hi = np.maximum.reduceat(boxes[:, 4:], starts, axis=0)
    gb = np.ascontiguousarray(np.concatenate([lo, hi], axis=1), np.float32)
    m = len(gb)
    nodes = np.zeros(2 * m - 1, L.NODE_DTYPE)
    order = np.zeros(m, np.uint32)
    nn, med = C.c_uint32(), C.c_uint32()
    assert L.lib().sr_bvh_build_host(gb.ctypes.data, m, 4, nodes.ctypes.data, len(nodes), order.ctypes.data, C.byref(nn),
                                     C.byref(med)) == L.SR_OK
    nodes = nodes[:nn.value].copy()
    # The groups' records in leaf order, and the leaf ranges in records.
    sizes = np.minimum(group, n - starts)[order]
    first = np.concatenate([[0], np.cumsum(sizes)])
    leaf = nodes["count"] > 0
    f, c = nodes["right_or_first"][leaf], nodes["count"][leaf]
    count = first[f + c] - first[f]
    assert count.max() <= 63
    nodes["right_or_first"][leaf], nodes["count"][leaf] = first[f], count
    slots = np.concatenate([np.arange(starts[g], min(starts[g] + group, n)) for g in order])
    engine.upload(BIG, sr.PackedScene(nodes, geoms[slots], attrs[slots], p.materials, p.stars, 0, p.light_pos, slots.astype(np.uint32)))
    seen = 0
    for pos in ((0.0, 0.0, 0.0, 0.0), (-20.0, 5.0, 3.0, -4.0), (-40.0, -10.0, 6.0, 2.0)):
        cam = sr.camera(pos, 110.0, rapidity=(0.4, 0.1, -0.3))
        u = sr.uniforms(cam, 203, 117, 0, 1, 0, num_nodes=len(nodes), light_pos=p.light_pos)
        seen += int((_both(engine, BIG, u, None).hit_id != 0xFFFFFFFF).sum())
    assert seen > 0


@pytest.mark.parametrize("side", [-2, 2])
def test_small_scene_either_side_of_the_line(engine, side):
    """36,864 records: their rays walk alone up to 2^36 / 36,864 pixels a launch, as packets from there on."""
    s = sr.synth_scene(1, 1, n_bodies=16)
    engine.build_tubes(BIG, s)
    edge = 2**36 / engine.stats(BIG).num_prims
    w, h = 1366, int(edge / 1366) + side
    assert (w * h < edge) == (side < 0)
    u, cam = _u(s, w, h, (0.3, -0.2, 0.4))
    assert (_both(engine, BIG, u, cam).hit_id != 0xFFFFFFFF).any()


def test_frames_of_growing_size_in_turn(engine, bodies):
    """What one frame's walks leave in the queue and the list of shadow rays must not reach the next frame,
    whatever its size (the lists are kept between frames)."""
    for w, h in ((96, 64), (320, 200), (200, 120), (640, 400), (96, 64), (800, 500)):
        u, cam = _u(bodies, w, h, (-0.9, 0.8, 1.0))
        _both(engine, IDX, u, cam)


@pytest.mark.parametrize("layout", [L.SR_LAYOUT_OCTANT, L.SR_LAYOUT_COMPACT])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 3000])
def test_caller_rays_on_the_node_layout(engine, bodies, layout, n):
    """sr_trace_rays walks the node layout for rays of a positive finite range and the reference's nodes for
    others: a ray cast alone, among others and in another block position has the same hit, and rays of
    odd ranges (zero, negative, endless) the hits of the same rays within that range."""
    engine.set_layout(IDX, layout)
    try:
        rng = np.random.default_rng(n)
        d = rng.normal(size=(n, 3))
        rays = np.zeros((n, 10))
        rays[:, 4], rays[:, 5:8] = -1.0, d / np.linalg.norm(d, axis=1, keepdims=True)
        rays[:, 8], rays[:, 9] = 1e-3, 180.0
        h = engine.trace_rays(IDX, rays)
        back = engine.trace_rays(IDX, rays[::-1])[::-1]
        assert h.tobytes() == back.tobytes()
        odd = rays.copy()
        odd[:, 8] = 0.0  # the reference's nodes: no geometry lies at the observer, so the same hits
        o = engine.trace_rays(IDX, odd)
        near = (o["lambda_"] != h["lambda_"]) & (o["lambda_"] < 1e-3)
        assert (o["slot"][~near] == h["slot"][~near]).all() and (o["lambda_"][~near] == h["lambda_"][~near]).all()
        odd[:, 8], odd[:, 9] = 1e-3, np.inf
        e = engine.trace_rays(IDX, odd)
        hit = h["slot"] != 0xFFFFFFFF
        assert (e["slot"][hit] == h["slot"][hit]).all()
        with pytest.raises(ValueError):
            engine.trace_rays(IDX, np.zeros((2, 1)))
    finally:
        engine.set_layout(IDX, L.SR_LAYOUT_AUTO)
