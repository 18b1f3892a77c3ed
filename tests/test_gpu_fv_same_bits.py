"""The three forms of the first-order update, the sweep of one patch or a patch
grid, the 32 x 8 tile kernel (tuning key 5 = 1) and the batch's sweep, write out
the same fused operations in the same order: equal bits, states and time steps,
whatever the strip heights, row blocks and patches per warp."""
import numpy as np
import pytest

import exahype_b200 as E
from exahype_b200 import DeviceBuffer, FVPatches

pytestmark = pytest.mark.gpu


def run(make, form, steps=3):
    E._lib.call('exa_tune_set', 5, form)
    try:
        g = make()
        g.init(amp=0.2, seed=33, noise=1e-2)
        g.step(steps)
        u, s = g.get_state(), g.status()
        u = g.interiors(u).copy() if hasattr(g, 'interiors') else g.interior(u).copy()
        g.destroy()
        return u, s['time'], s.get('dt_next')
    finally:
        E._lib.call('exa_tune_set', 5, 0)


@pytest.mark.parametrize('pde', [E.PDE_EULER, E.PDE_EULER_PLANAR])
@pytest.mark.parametrize('size', [3, 31, 64, 121, 257, 701, 2051])
def test_sweep_and_tiles(size, pde):
    (a, ta, da), (b, tb, db) = (run(lambda: E.FVGrid(0, size, pde=pde), f) for f in (1, 0))
    assert np.array_equal(a, b) and ta == tb and da == db


@pytest.mark.parametrize('patch,npx,npy,bc', [(4, 1, 3, (0, 0)), (10, 31, 2, (1, 2)), (7, 40, 60, (0, 0)),
                                              (25, 30, 41, (2, 1))])
def test_patch_grids(patch, npx, npy, bc):
    def make():
        g = E.FVPatchGrid(0, patch, npx, npy)
        g.set_boundary(bc)
        return g

    (a, ta, da), (b, tb, db) = (run(make, f) for f in (1, 0))
    assert np.array_equal(a, b) and ta == tb and da == db


@pytest.mark.parametrize('pde', [E.PDE_EULER, E.PDE_EULER_PLANAR])
@pytest.mark.parametrize('size', [2, 7, 10, 14, 15, 29, 30, 31, 33, 64, 100])
def test_batch_and_sweep(size, pde):
    g = E.FVGrid(0, size, pde=pde)
    g.init(amp=0.2, seed=34, noise=1e-2)
    u = g.get_state()
    g.step(1)
    want, dt = g.interior().copy(), g.status()['time']
    g.destroy()
    for n in (1, 40, 3000 if size < 20 else 60):
        k = FVPatches(size, 1, [1.0, 1.0], pde=pde)
        old = DeviceBuffer.from_array(np.tile(u, n))
        k.periodic_ghosts(n, old)
        new = DeviceBuffer.from_array(old.download())
        k.godunov_update(n, new, old, dt)
        got = new.download().reshape(n, size + 2, size + 2, 5)[:, 1:-1, 1:-1]
        assert np.array_equal(got, np.broadcast_to(want, got.shape))
