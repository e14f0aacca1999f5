"""The bloom's coarse levels, taken by one block per observer up to 1024 pixels a level: frames on either side of that
line, and batches whose observers lie on both, equal the plain path's."""
import numpy as np
import pytest

import specrel_b200 as sr

pytestmark = pytest.mark.gpu

IDX = 46
# Level 3 of 256x256 has 32x32 pixels; the others are a row or column off it, one pixel wide, or past it at level 5.
SIZES = [(256, 256), (257, 256), (256, 249), (248, 264), (2049, 33), (1, 1025), (1024, 1), (1025, 1), (1024, 1024), (3, 2)]


@pytest.fixture(scope="module")
def scene(engine):
    s = sr.synth_scene(1, 1, n_bodies=8)
    engine.build_tubes(IDX, s)
    return s


def _u(scene, w, h):
    return sr.uniforms(sr.camera((-20.0, 0.0, 0.0, -6.0), 80.0, rapidity=(0.2, 0.1, -0.3)), w, h, 0, 1, 0,
                       num_nodes=scene.num_nodes, light_pos=scene.light_pos)


@pytest.mark.parametrize("size", SIZES)
def test_single_frames(engine, scene, size):
    u = _u(scene, *size)
    assert (engine.render(IDX, u).rgb == engine.render(IDX, u, path=sr.SR_PATH_PLAIN).rgb).all()


def test_batches_on_both_sides(engine, scene):
    us = [_u(scene, w, h) for w, h in SIZES]
    out = np.zeros(sum(w * h for w, h in SIZES), np.uint32)
    for order in (us, us[::-1], us[:2] + us[-1:]):
        n = sum(u.size[0] * u.size[1] for u in order)
        engine.render_batch(IDX, order, out.ctypes.data, n, device_output=False)
        off = 0
        for u in order:
            k = u.size[0] * u.size[1]
            assert (out[off:off + k] == engine.render(IDX, u, path=sr.SR_PATH_PLAIN).rgb).all()
            off += k
