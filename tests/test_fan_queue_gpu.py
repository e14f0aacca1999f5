"""The packet walk's queue (sr_fast.cu): tiles, groups and single shadow queries that are given up really pass
through it, and a wait in it that runs out leaves an error behind, not entries that a later frame takes as its own."""
import ctypes as C

import numpy as np
import pytest
import torch

import specrel_b200 as sr
from specrel_b200 import _lib as L

pytestmark = pytest.mark.gpu

POLLS = 1 << 21  # FastCtx::fan_polls


@pytest.fixture(scope="module")
def world():
    eng = sr.Engine(0)
    scene = sr.synth_scene(2, 3, n_bodies=8)
    eng.build_tubes(0, scene)
    yield eng, scene
    eng.close()


def _polls(eng, n):
    f = L.lib().sr_test_queue_polls
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32], C.c_int
    assert f(eng.h, n) == 0


def _queued(eng):
    f = L.lib().sr_test_queued
    f.argtypes, f.restype = [C.c_void_p, C.POINTER(C.c_uint32)], C.c_int
    out = (C.c_uint32 * 2)()
    assert f(eng.h, out) == 0
    return list(out)


def _view(scene, w, h, rapidity=(1.6, -1.4, 1.2), fov=150.0, shadow=1):
    pos = (0.0, 0.0, 0.0, 0.0)
    return (sr.uniforms(sr.camera(pos, fov, rapidity=rapidity), w, h, 0, shadow, 0, num_nodes=scene.num_nodes,
                        light_pos=scene.light_pos), sr.cam64(pos, rapidity))


def _exact(eng, u, cam):
    keep = eng.tuning(0)
    got = eng.render(0, u, aux=True, cam=cam)
    queued = _queued(eng)
    t = eng.tuning(0)
    t.packet = 0
    eng.set_tuning(0, t)
    try:
        ref = eng.render(0, u, aux=True, cam=cam)
    finally:
        eng.set_tuning(0, keep)
    assert (got.hit_id == ref.hit_id).all() and (got.rgb == ref.rgb).all()
    assert (got.lam.view(np.uint32) == ref.lam.view(np.uint32)).all()
    return np.array(queued + [(ref.hit_id != 0xFFFFFFFF).sum()])


@pytest.mark.parametrize("w,h", [(95, 41), (471, 163), (640, 400)])
def test_wide_views_pass_through_the_queue(world, w, h):
    """Tiles given up are walked in groups, groups in pairs, and shadow walks given up query by query."""
    eng, scene = world
    total = np.zeros(3, int)
    for rapidity in ((1.6, -1.4, 1.2), (-2.0, 1.0, -2.0), (-0.9, 0.8, 1.0)):
        for fov in (60.0, 150.0):
            total += _exact(eng, *_view(scene, w, h, rapidity, fov))
    print("queued in the two launches, and hits:", total)
    assert (total > 0).all()


def test_a_wait_that_runs_out_is_reported_and_leaves_nothing_behind(world):
    eng, scene = world
    views = [_view(scene, w, h) for w, h in ((640, 400), (471, 163), (95, 41), (320, 200))]
    out = torch.zeros(640 * 400, dtype=torch.int32, device="cuda")
    assert _exact(eng, *views[0])[0] > 0
    eng.synchronize()
    ran_out = 0
    for u, cam in views:
        _polls(eng, 0)
        try:
            eng.render(0, u, aux=True, cam=cam)
        except sr.SrError as e:
            assert e.status == L.SR_ERR_CUDA
            ran_out += 1
        finally:
            _polls(eng, POLLS)
        for v, c in views:  # every frame after it is exact, larger and smaller ones
            _exact(eng, v, c)
        eng.synchronize()  # reported once
    assert ran_out > 0
    # A frame that stays on the device returns before its flags are there: the next call that waits reports.
    _polls(eng, 0)
    try:
        for u, cam in views:
            eng.render_into(0, u, out.data_ptr(), cam=cam)
    finally:
        _polls(eng, POLLS)
    with pytest.raises(sr.SrError):
        eng.synchronize()
    eng.synchronize()
    for u, cam in views:
        _exact(eng, u, cam)


def test_engines_in_turn(world):
    """Three engines' packet frames and batches queued one after the other without a wait between them: each engine's
    launches may run beside another's, whose waiting warps must not keep them from their work."""
    _, scene = world
    engines = [sr.Engine(0) for _ in range(3)]
    try:
        views = [[_view(scene, w, h, rapidity=r) for w, h in ((640, 400), (95, 41), (320, 200))]
                 for r in ((1.6, -1.4, 1.2), (-0.9, 0.8, 1.0), (0.3, -0.2, 0.4))]
        n = sum(u.size[0] * u.size[1] for u, _ in views[0])
        outs = [[torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(8)] for _ in engines]
        for e in engines:
            e.build_tubes(0, scene)
        for turn in range(8):
            for e, v, o in zip(engines, views, outs):
                e.render_batch(0, [u for u, _ in v], o[turn].data_ptr(), n, cams=[c for _, c in v])
                e.render_into(0, v[1][0], o[turn].data_ptr() + 4 * 640 * 400, cam=v[1][1])
        for e, v, o in zip(engines, views, outs):
            e.synchronize()
            t = e.tuning(0)
            t.packet = 0
            e.set_tuning(0, t)
            ref = np.zeros(n, np.uint32)
            e.render_batch(0, [u for u, _ in v], ref.ctypes.data, n, cams=[c for _, c in v], device_output=False)
            for x in o:
                assert (x.cpu().numpy().view(np.uint32) == ref).all()
    finally:
        for e in engines:
            e.close()
