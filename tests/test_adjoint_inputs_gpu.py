"""What a gradient call (sr_adjoint) reads: the forward frame's star lists up to the room that frame had, and the
caller's target image wherever it lies."""
import ctypes as C

import numpy as np
import pytest
import torch

import specrel_b200 as sr
from specrel_b200 import _lib as L

pytestmark = pytest.mark.gpu

W, H = 160, 100
AT, FROM = (0.0, 0.0, 0.0, 0.0), (0.75, -0.25, 0.45)


@pytest.fixture(scope="module")
def scene():
    return sr.synth_scene(5, 2, n_bodies=8, steps=16, n_stars=2000)


def _engine(scene, room=0):
    eng = sr.Engine(0)
    eng.build_tubes(0, scene)
    f = L.lib().sr_test_star_room
    f.argtypes, f.restype = [C.c_void_p, C.c_uint32], C.c_int
    assert f(eng.h, room) == 0
    return eng


def _uniforms(scene, w=W, h=H):
    return sr.uniforms(sr.camera(AT, 90.0), w, h, 0, 1, 0, num_nodes=scene.num_nodes, num_stars=scene.num_stars)


def _target(eng, scene):
    return torch.tensor(eng.render(0, _uniforms(scene), hdr=True, cam=sr.cam64(AT, (0.8, -0.3, 0.5))).hdr).cuda()


def _values(r):
    return [r.loss, r.primal_mismatch, r.star_terms] + list(r.grad)


@pytest.mark.parametrize("room", [1, 300, 1000])
def test_lists_longer_than_their_room_after_a_larger_batch(scene, room):
    """A batch of more observers leaves a larger list buffer behind: the tiles whose lists the gradient's own
    frame had no room for are summed without lists all the same, as in a fresh context."""
    u, cam = _uniforms(scene), sr.cam64(AT, FROM)
    fresh, used = _engine(scene, room), _engine(scene, room)
    try:
        us = [_uniforms(scene, 320, 200) for _ in range(6)]
        out = np.zeros(6 * 320 * 200, np.uint32)
        used.render_batch(0, us, out.ctypes.data, out.size, cams=[sr.cam64(AT, (-0.2, 0.1 * k, 0.3)) for k in range(6)],
                          device_output=False)
        target = _target(fresh, scene)
        for level in (0, 3):
            a, b = (_values(e.adjoint(0, u, cam, target.data_ptr(), level=level)) for e in (fresh, used))
            assert a == b
            assert a[1] > 0  # pixels of such tiles are counted
    finally:
        fresh.close()
        used.close()


@pytest.mark.parametrize("level", [0, 3])
def test_target_at_any_float_address(scene, level):
    """The target is width * height * 4 floats: a view that starts at an odd float gives the same loss and
    gradient, frozen evaluations too."""
    u, cam = _uniforms(scene), sr.cam64(AT, FROM)
    eng = _engine(scene)
    try:
        target = _target(eng, scene)
        ref = _values(eng.adjoint(0, u, cam, target.data_ptr(), level=level))
        frozen = eng.adjoint(0, u, cam, target.data_ptr(), level=level, frozen=True).loss
        room = torch.zeros(4 * W * H + 8, device="cuda")
        for shift in (1, 2, 3, 5):
            view = room[shift:shift + 4 * W * H]
            view.copy_(target.reshape(-1))
            assert view.data_ptr() % 16 != 0
            assert _values(eng.adjoint(0, u, cam, view.data_ptr(), level=level)) == ref
            assert eng.adjoint(0, u, cam, view.data_ptr(), level=level, frozen=True).loss == frozen
        assert _values(eng.adjoint(0, u, cam, target.data_ptr(), level=level)) == ref
    finally:
        eng.close()
