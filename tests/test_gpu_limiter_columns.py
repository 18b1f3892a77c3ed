"""Limiter kernels where their splits can go wrong: single cells, partial last
CTAs, batches on both sides of the size rules (whole patches or streamed planes
in FV -> DG, columns or whole 2D cells in the extrema), variable counts other
than five, fewer observables than variables.

A projected value is DIM nested sums of at most 13 products (39 roundings of
1.1e-16) of values of one size with weights whose absolute sums stay below about
10 (FV -> DG, order 6): 1e-13 of the largest value.  A batch's cells and the same
cells alone take the same fused multiply-adds in the same order: equal bits."""
import numpy as np
import pytest

import _oracle as O
from exahype_b200 import DeviceBuffer, limiter

pytestmark = pytest.mark.gpu
TOL = 1e-13


def data(dim, order, cells, nvar, ghost, seed):
    rng = np.random.default_rng(seed)
    s = O.lim_sizes(dim, order, nvar, ghost)
    return s, rng.uniform(0.5, 4.0, cells * s['luh']), rng.uniform(0.5, 4.0, cells * s['lim'])


def run(dim, order, cells, nvar, nobs, ghost, luh, lim):
    d_luh, d_lim = DeviceBuffer.from_array(luh), DeviceBuffer.from_array(np.full_like(lim, -7.0))
    d_in, d_back = DeviceBuffer.from_array(lim), DeviceBuffer(luh.size)
    nb = cells * 2 * dim * nobs
    d_mn, d_mx = DeviceBuffer(nb), DeviceBuffer(nb)
    limiter.project_on_fv(dim, order, cells, d_luh, d_lim, nvar=nvar, ghost=ghost)
    limiter.project_on_dg(dim, order, cells, d_in, d_back, nvar=nvar, ghost=ghost)
    limiter.local_min_max(dim, order, cells, d_luh, d_mn, d_mx, nvar=nvar, nobs=nobs)
    return [b.download().reshape(cells, -1) for b in (d_lim, d_back, d_mn, d_mx)]


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('order', [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize('cells,nvar,nobs,ghost', [(1, 5, 5, 2), (7, 1, 1, 0), (3, 4, 2, 1), (601, 5, 3, 1),
                                                   (1203, 5, 5, 2)])
def test_columns_vs_oracle(dim, order, cells, nvar, nobs, ghost):
    s, luh, lim = data(dim, order, cells, nvar, ghost, 100 * dim + 10 * order + cells)
    fv, dg, mn, mx = run(dim, order, cells, nvar, nobs, ghost, luh, lim)
    pick = [0, cells // 2, cells - 1]
    for c in pick:
        u, l = luh.reshape(cells, -1)[c], lim.reshape(cells, -1)[c]
        ref = O.limiter_project_on_fv(dim, order, u, nvar=nvar, ghost=ghost, lim=np.full(l.size, -7.0))
        assert np.abs(fv[c] - ref.ravel()).max() <= TOL * np.abs(ref).max(), c
        ref = O.limiter_project_on_dg(dim, order, l, nvar=nvar, ghost=ghost)
        assert np.abs(dg[c] - ref.ravel()).max() <= TOL * np.abs(ref).max(), c
        rmn, rmx = O.limiter_local_min_max(dim, order, u, nvar=nvar, nobs=nobs)
        assert np.abs(mn[c] - rmn.ravel()).max() <= TOL * np.abs(rmn).max(), c
        assert np.abs(mx[c] - rmx.ravel()).max() <= TOL * np.abs(rmx).max(), c


@pytest.mark.parametrize('dim,order,cells', [(2, 1, 40001), (2, 3, 16001), (2, 4, 16001), (2, 5, 16001), (3, 2, 25001),
                                             (3, 4, 6701), (3, 5, 3801)])
def test_large_batch_equals_its_cells_alone(dim, order, cells):
    s, luh, lim = data(dim, order, cells, 5, 1, order)
    big = run(dim, order, cells, 5, 5, 1, luh, lim)
    for lo, n in ((0, 5), (cells - 130, 130)):
        few = run(dim, order, n, 5, 5, 1, luh.reshape(cells, -1)[lo:lo + n].ravel().copy(),
                  lim.reshape(cells, -1)[lo:lo + n].ravel().copy())
        for a, b in zip(big, few):
            assert np.array_equal(a[lo:lo + n], b)
