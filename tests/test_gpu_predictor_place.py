"""A cell's predictor result does not depend on where the cell lies in the
call: its place in a block decides which lanes and warps add up its residual,
and the sum of the rounded squares must not depend on that when it is compared
with the tolerance.

The states are scaled so that the first residual lies within a few units in
the last place of the tolerance (the Euler equations are homogeneous in the
state: scaled by s, the residual scales by s^2, and its own roundings stay
relative to it).  Then one unit of s decides whether a cell takes one iteration
or two, and so does one unit in the sum."""
import numpy as np
import pytest

import exahype_b200 as E
from exahype_b200 import DeviceBuffer

pytestmark = pytest.mark.gpu
V = 5
DX, DT = [0.05, 0.04], 3e-3


def predict(variant, order, q, pde=E.PDE_EULER):
    """q [cell][node][V] -> outputs and iterations per cell (tuning key 3 = variant)"""
    cells, B = q.shape[0], order + 1
    k = E.BatchedADERDG(2, order, DX, pde=pde)
    out = [DeviceBuffer(cells * n * V) for n in (B * B, 4 * B, 4 * B)]
    it = DeviceBuffer(cells, np.int32)
    E._lib.call('exa_tune_set', 3, variant)
    try:
        k.predictor_vi(cells, DeviceBuffer.from_array(q.ravel()), DT, *out, iters=it)
        return [b.download().reshape(cells, -1) for b in out], it.download()
    finally:
        E._lib.call('exa_tune_set', 3, 0)


def rough_cells(order, cells, seed):
    rng = np.random.default_rng(seed)
    nn = (order + 1) ** 2
    q = np.zeros((cells, nn, V))
    q[..., 0] = 1.0 + 0.1 * rng.random((cells, nn))
    q[..., 1:4] = 0.1 * rng.standard_normal((cells, nn, 3))
    q[..., 4] = 2.5 + 0.1 * rng.random((cells, nn))
    return q


def threshold_scales(variant, order, q):
    """per cell the largest s (to the last bit) with which s * q takes one iteration"""
    lo, hi = np.full(len(q), 1e-12), np.ones(len(q))
    for _ in range(200):
        mid = lo + 0.5 * (hi - lo)
        if ((mid == lo) | (mid == hi)).all():
            break
        one = predict(variant, order, mid[:, None, None] * q)[1] == 1
        lo, hi = np.where(one, mid, lo), np.where(one, hi, mid)
    assert (predict(variant, order, lo[:, None, None] * q)[1] == 1).all()
    assert (predict(variant, order, hi[:, None, None] * q)[1] > 1).all()
    return lo


def around(s, ulps):
    for _ in range(abs(ulps)):
        s = np.nextafter(s, np.inf if ulps > 0 else 0.0)
    return s


@pytest.mark.parametrize('order,variant', [(2, 4), (3, 4), (4, 4), (5, 4), (2, 0), (5, 0)])
def test_every_place_stops_alike(order, variant):
    contents, places = 200, 32
    q = rough_cells(order, contents, 17 + order)
    s = threshold_scales(variant, order, q)
    iters = set()
    for ulps in range(-6, 7):
        u = around(s, ulps)[:, None, None] * q
        out, it = predict(variant, order, np.repeat(u, places, axis=0))
        it = it.reshape(contents, places)
        assert (it == it[:, :1]).all(), (ulps, int((it != it[:, :1]).any(axis=1).sum()))
        for o in out:
            o = o.reshape(contents, places, -1)
            assert np.array_equal(o, np.broadcast_to(o[:, :1], o.shape))
        iters |= set(it.ravel())
    assert len(iters) > 1
