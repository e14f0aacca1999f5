"""Trees whose splits peel a few primitives off at a time, built on the device (sr_build_scene): a subtree of 2048
primitives or fewer that would have more than 64 nodes waiting in one block's depth-first build is refused, whichever
way it is built; one whose nodes wait on the other side is not, and every tree that is built is the host's."""
import ctypes as C

import numpy as np
import pytest

import specrel_b200 as sr
from specrel_b200 import _lib as L

pytestmark = pytest.mark.gpu

IDX = 49


def _chain(m, ratio, axes, far, sign=1.0):
    """m boxes a geometric step apart along each of `axes` axes in turn, and `far` boxes beyond them."""
    step = 1e-3 * ratio ** np.arange(m)
    rng = np.random.default_rng(m)
    rows = [np.zeros((m, 4)) for _ in range(axes)]
    for a in range(axes):
        rows[a][:, a] = step
    beyond = np.zeros((far, 4))
    beyond[:, 0] = step[-1] * 1e3 * (30.0 + 0.01 * np.arange(far))
    c = np.concatenate(rows + [beyond])
    c[:, 2:] += rng.normal(size=(len(c), 2)) * 1e-4
    c = (sign * c).astype(np.float32)
    return np.ascontiguousarray(np.concatenate([c - np.float32(1e-5), c + np.float32(1e-5)], 1))


def _build(engine, b):
    mats = sr.synth_scene(1, 1, n_bodies=2, steps=2).packed().materials
    engine.build(IDX, b, np.zeros(len(b), sr.GEOM_DTYPE), np.zeros(len(b), sr.ATTR_DTYPE), mats)


def _host(b):
    nodes, order = np.zeros(2 * len(b), L.NODE_DTYPE), np.zeros(len(b), np.uint32)
    nn, med = C.c_uint32(), C.c_uint32()
    assert L.lib().sr_bvh_build_host(b.ctypes.data, len(b), 4, nodes.ctypes.data, len(nodes), order.ctypes.data,
                                     C.byref(nn), C.byref(med)) == L.SR_OK
    assert med.value == 0
    return nodes[:nn.value], order


@pytest.mark.parametrize("m,ratio,axes,far", [(900, 1.08, 1, 8000), (1000, 1.03, 2, 8000), (600, 1.06, 1, 7000), (400, 1.15, 1, 8000)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_peeled_trees_are_the_hosts(engine, m, ratio, axes, far, sign):
    b = _chain(m, ratio, axes, far, sign)
    _build(engine, b)
    nodes, order = engine.tree(IDX)
    hn, ho = _host(b)
    assert nodes.tobytes() == hn.tobytes() and (order == ho).all()


@pytest.mark.parametrize("far", [0, 7000, 8000])  # alone in a block, and below and above the line of the warp build
@pytest.mark.parametrize("m,ratio", [(400, 1.15), (900, 1.08)])
def test_trees_too_deep_are_refused(engine, m, ratio, far):
    with pytest.raises(sr.SrError) as e:
        _build(engine, _chain(m, ratio, 2, far))
    assert e.value.status == L.SR_ERR_UNSUPPORTED
