"""Slabs on one side of the size where the 2D predictor of orders 2 and 5
changes its form and their undivided grid on the other (8 cells per SM at order
2, 4 at order 5; 1184 and 592 with 148 SMs), and on the same side: the slabs
equal the undivided grid bit for bit all the same."""
import numpy as np
import pytest

import exahype_b200 as E
from exahype_b200 import slab as SL

pytestmark = pytest.mark.gpu
IC = dict(kind=0, param=5.0, seed=3, noise=1e-3)


@pytest.mark.parametrize('order,n,world', [
    (2, (40, 40), 4), (2, (36, 36), 2), (2, (30, 60), 3), (2, (7, 9), 3), (3, (25, 32), 4),
    (5, (40, 40), 4), (5, (24, 48), 2), (5, (25, 27), 9), (5, (7, 9), 3)])
def test_slabs_equal_undivided_grid(order, n, world):
    steps = 3
    g = E.ADERDGGrid(2, order, n)
    g.init(**IC)
    g.step(steps)
    ref, t = g.get_state(), g.status()['time']
    g.destroy()
    slabs = [SL.SlabGrid(2, order, n, r, world) for r in range(world)]
    for s in slabs:
        s.init(**IC)
    ring = SL.LocalRing(slabs)
    SL.prime(ring)
    SL.step(ring, None, steps)
    got = SL.gather_state(slabs)
    for s in slabs:
        assert s.status()['time'] == t
        s.destroy()
    assert np.array_equal(got, ref)
