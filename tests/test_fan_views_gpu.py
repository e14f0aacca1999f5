"""Views past 180 degrees: the image plane's half extents are negative there (tan of half the angle), and the
packet walk's bounds must hold the rays all the same."""
import numpy as np
import pytest

import specrel_b200 as sr

pytestmark = pytest.mark.gpu

CUBES = 44


@pytest.fixture(scope="module")
def cubes(engine):
    s = sr.synth_scene(1, 5, n_bodies=64)  # too large for the lone walk
    engine.build_tubes(CUBES, s)
    return s


@pytest.mark.parametrize("slice_mode", [0, 1, 2])
@pytest.mark.parametrize("fov", [120.0, 179.0, 181.0, 190.0, 200.0, 270.0, 340.0])
def test_frames_equal_the_plain_path(engine, cubes, fov, slice_mode):
    for pos in ((0.0, 0.0, 0.0, 0.0), (-20.0, 5.0, 3.0, -4.0), (-40.0, -10.0, 6.0, 2.0)):
        u = sr.uniforms(sr.camera(pos, fov, rapidity=(0.4, 0.1, -0.3)), 640, 400, 0, 1, slice_mode,
                        num_nodes=cubes.num_nodes, light_pos=cubes.light_pos)
        assert (u.half_wh[0] < 0.0) == (fov > 180.0)
        a, b = (engine.render(CUBES, u, path=path, aux=True) for path in (sr.SR_PATH_FAST, sr.SR_PATH_PLAIN))
        assert (a.hit_id == b.hit_id).all() and (a.lam.view(np.uint32) == b.lam.view(np.uint32)).all()
        assert (a.rgb == b.rgb).all()
