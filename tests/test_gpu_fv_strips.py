"""The Godunov sweep at sizes that give its strips different heights (rows and
columns that do not divide, one strip or many, the height's line between 31 and
32 rows) against the 32 x 8 tile kernel (tuning key 5 = 1).

Both perform the same operations; a multiply-add may be contracted in one and
not in the other, one rounding of 1.1e-16 per operation and some twenty
operations per step along a value's path: 1e-14 relative after three steps."""
import numpy as np
import pytest

import exahype_b200 as E

pytestmark = pytest.mark.gpu


def run(make, form):
    E._lib.call('exa_tune_set', 5, form)
    try:
        g = make()
        g.init(amp=0.2, seed=21, noise=1e-3)
        g.step(3)
        u, t = g.get_state(), g.status()['time']
        u = g.interiors(u).copy() if hasattr(g, 'interiors') else u.copy()
        g.destroy()
        return u.ravel(), t
    finally:
        E._lib.call('exa_tune_set', 5, 0)


@pytest.mark.parametrize('size', [8, 31, 64, 121, 257, 370, 513, 701, 1025, 1500, 2051])
def test_strip_heights_patch(size):
    def interior(u):
        s = int(round((u.size // 5) ** 0.5))
        return u.reshape(s, s, 5)[1:-1, 1:-1]
    (a, ta), (b, tb) = (run(lambda: E.FVGrid(0, size), f) for f in (1, 0))
    a, b = interior(a), interior(b)
    assert np.linalg.norm(a - b) <= 1e-14 * np.linalg.norm(a)
    assert abs(ta - tb) <= 1e-14 * ta


@pytest.mark.parametrize('patch,npx,npy', [(4, 1, 3), (10, 31, 2), (7, 40, 60), (25, 30, 41)])
def test_strip_heights_grid(patch, npx, npy):
    (a, ta), (b, tb) = (run(lambda: E.FVPatchGrid(0, patch, npx, npy), f) for f in (1, 0))
    assert np.linalg.norm(a - b) <= 1e-14 * np.linalg.norm(a)
    assert abs(ta - tb) <= 1e-14 * ta
