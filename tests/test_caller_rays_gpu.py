"""Caller rays (sr_trace_rays) by every route: a warp per ray over the fan layout, a thread per ray for long lists and
for the rays that the layout does not take. The reference's own walk answers a ray scaled by a power of two past
the layouts' range of values: its hit is the ray's, divided."""
import numpy as np
import pytest

import specrel_b200 as sr
from test_packet_gpu import tie_scene

pytestmark = pytest.mark.gpu

IDX, TIES = 47, 48
UP = 2.0 ** 41
LONG = 1 << 16  # RAYS_LONG


@pytest.fixture(scope="module")
def bodies(engine):
    s = sr.synth_scene(2, 3, n_bodies=8)
    engine.build_tubes(IDX, s)
    return s


def _rays(seed, n, t_min=1e-3, t_max=180.0, at=(0.0, 0.0, 0.0, 0.0)):
    d = np.random.default_rng(seed).normal(size=(n, 3))
    rays = np.zeros((n, 10))
    rays[:, 0:4], rays[:, 4], rays[:, 5:8] = at, -1.0, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 8], rays[:, 9] = t_min, t_max
    return rays.astype(np.float32).astype(np.float64)


def _reference(engine, idx, rays):
    far = rays.copy()
    far[:, 4:8] *= UP
    far[:, 8:10] /= UP
    h = engine.trace_rays(idx, far)
    return h["slot"], h["lambda_"] * np.float32(UP)


def _check(engine, idx, rays):
    slot, lam = _reference(engine, idx, rays)
    h = engine.trace_rays(idx, rays)
    assert (h["slot"] == slot).all() and (h["lambda_"] == lam).all()
    assert (slot != 0xFFFFFFFF).any()
    return h


@pytest.mark.parametrize("t_min", [0.0, -0.0, 1e-30, 1e-3, 5.0])
def test_ranges_from_zero_on(engine, bodies, t_min):
    _check(engine, IDX, _rays(1, 4000, t_min))


def test_rays_that_start_inside_bodies(engine, bodies):
    """From events where bodies are: entries at 0, and boxes entered before the range begins."""
    inside = _rays(2, 2000)
    hit = engine.trace_rays(IDX, inside)
    ev = hit["event"][hit["slot"] != 0xFFFFFFFF][:40]
    assert len(ev) > 10
    for k, at in enumerate(ev[::5]):
        for t_min in (0.0, 1e-3):
            _check(engine, IDX, _rays(3 + k, 500, t_min, at=at))


@pytest.mark.parametrize("n", [LONG - 1, LONG, LONG + 1])
def test_lists_on_both_sides_of_the_line(engine, bodies, n):
    rays = _rays(4, n)
    rays[::3, 8] = 0.0
    h = _check(engine, IDX, rays)
    part = engine.trace_rays(IDX, rays[n - 300:])
    assert part.tobytes() == h[n - 300:].tobytes()


@pytest.mark.parametrize("n", [3000, 1 << 14, (1 << 14) + 1])  # walked by their warps, and listed
def test_rays_the_layout_does_not_take_among_others(engine, bodies, n):
    """Negative and NaN ranges, endless ones and values beyond 1e12, scattered over a list: every ray has the hit it
    has alone, and the list's order does not matter."""
    rays = _rays(5, n)
    odd = {0: (8, -1.0), 5: (8, np.nan), 11: (9, np.inf), 17: (9, 0.0), 23: (0, 1e13), 29: (9, np.nan), 31: (9, -1.0)}
    for k, (col, v) in odd.items():
        rays[k::97, col] = v
    h = engine.trace_rays(IDX, rays)
    assert engine.trace_rays(IDX, rays[::-1])[::-1].tobytes() == h.tobytes()
    for k in list(odd) + [1, 2, 3]:
        assert engine.trace_rays(IDX, rays[k:k + 1]).tobytes() == h[k:k + 1].tobytes()
    kept = np.ones(len(rays), bool)
    for k in odd:
        kept[k::97] = False
    slot, lam = _reference(engine, IDX, rays[kept])
    assert (h["slot"][kept] == slot).all() and (h["lambda_"][kept] == lam).all()


def test_equal_lambda_hits(engine):
    packed, n = tie_scene()
    engine.upload(TIES, packed)
    for at in ((0.0, 0.0, 0.0, 0.0), (-20.0, 5.0, 3.0, -4.0)):
        h = _check(engine, TIES, _rays(6, 4000, 0.0, at=at))
        ids = h["id"][h["slot"] != 0xFFFFFFFF]
        assert (ids >= n).any() and (ids < n).any()


@pytest.mark.parametrize("shape", [(3, 1), (2, 4), (2, 8), (2, 9), (2, 10, 1)])
def test_rays_of_too_few_values_are_refused(engine, bodies, shape):
    with pytest.raises(ValueError):
        engine.trace_rays(IDX, np.zeros(shape))
