"""The limiter's batched operators choose their kernel by the number of cells
and variables (passes through shared memory for few columns, register columns
for many; whole patches or streamed planes): a cell's result is the same bits
in all of them, whatever the batch, and the oracle's to 1e-12 relative (sums of
at most 13^3 products of O(1) tables and values)."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
from exahype_b200 import DeviceBuffer, limiter

pytestmark = pytest.mark.gpu
KINDS = 7


def counts(patch):
    """on both sides of the rules, as far as 130 MB of patches go"""
    return [KINDS] + [n for n in (200, 700, 900, 4000, 12000, 30000) if n * patch <= 1.6e7]


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('order', [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize('nvar,nobs,ghost', [(5, 5, 1), (1, 1, 2), (7, 3, 0)])
def test_cell_same_in_any_batch(dim, order, nvar, nobs, ghost):
    rng = np.random.default_rng(1000 * dim + 100 * order + nvar)
    nn, npt = (order + 1) ** dim, (2 * order + 1 + 2 * ghost) ** dim
    luh = 1.0 + rng.random((KINDS, nn * nvar))
    luh[3, nn // 2 * nvar] = np.nan  # (every sum over the cell; the other nodes stay)
    luh[4, (nn - 1) * nvar] = np.inf
    patch = 1.0 + rng.random((KINDS, npt * nvar))
    lo = 0.9 + 0.4 * rng.random((KINDS, 2 * dim * nobs))
    hi = 1.6 + 0.6 * rng.random((KINDS, 2 * dim * nobs))
    first = None
    for n in counts(npt * nvar):
        which = np.arange(n) % KINDS
        u, q = DeviceBuffer.from_array(luh[which].ravel()), DeviceBuffer.from_array(patch[which].ravel())
        lim, back = DeviceBuffer(n * npt * nvar), DeviceBuffer(n * nn * nvar)
        lim.zero()
        mn, mx = DeviceBuffer(n * 2 * dim * nobs), DeviceBuffer(n * 2 * dim * nobs)
        bmn, bmx = DeviceBuffer.from_array(lo[which].ravel()), DeviceBuffer.from_array(hi[which].ravel())
        fmn, fmx, ok = DeviceBuffer(mn.n), DeviceBuffer(mn.n), DeviceBuffer(n, np.int32)
        limiter.project_on_fv(dim, order, n, u, lim, nvar=nvar, ghost=ghost)
        limiter.project_on_dg(dim, order, n, q, back, nvar=nvar, ghost=ghost)
        limiter.local_min_max(dim, order, n, u, mn, mx, nvar=nvar, nobs=nobs)
        limiter.fv_min_max(dim, order, n, q, fmn, fmx, nvar=nvar, nobs=nobs, ghost=ghost)
        limiter.dmp(dim, order, n, u, bmn, bmx, ok, 1e-4, 1e-3, nvar=nvar, nobs=nobs)
        got = [b.download().reshape(n, -1) for b in (lim, back, mn, mx, fmn, fmx, bmn, bmx, ok)]
        if first is None:
            first = got
            check_oracle(dim, order, nvar, nobs, ghost, luh, patch, lo, hi, got)
        for a, b in zip(got, first):
            assert np.array_equal(a, b[which], equal_nan=True)


def check_oracle(dim, order, nvar, nobs, ghost, luh, patch, lo, hi, got):
    for c in (0, KINDS - 1):
        u, q = luh[c].copy(), patch[c].copy()
        ref = [O.limiter_project_on_fv(dim, order, u, nvar=nvar, ghost=ghost),
               O.limiter_project_on_dg(dim, order, q, nvar=nvar, ghost=ghost),
               *O.limiter_local_min_max(dim, order, u, nvar=nvar, nobs=nobs),
               *O.limiter_fv_min_max(dim, order, q, nvar=nvar, nobs=nobs, ghost=ghost)]
        for a, b in zip(got, ref):
            assert np.abs(a[c] - np.ravel(b)).max() <= 1e-12 * np.abs(b).max()
        ok, mn, mx = O.limiter_dmp(dim, order, u, lo[c].copy(), hi[c].copy(), 1e-4, 1e-3, nvar=nvar, nobs=nobs)
        assert bool(got[8][c][0]) == bool(np.ravel(ok)[0])
        assert np.abs(got[6][c] - np.ravel(mn)).max() <= 1e-12 * np.abs(mn).max()
        assert np.abs(got[7][c] - np.ravel(mx)).max() <= 1e-12 * np.abs(mx).max()
