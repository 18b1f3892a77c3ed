"""The space-time pencil predictor (the FP64 default) against the node-gather
predictor (tuning key 3 = 1) and the oracle, where it can go wrong: CTAs that
hold several cells with a partial last one, one cell alone, cells of one CTA
that need different iteration counts, both PDE forms.

Both kernels evaluate the same sums in another order.  A value is a sum of
about B (time) x DIM x B products of O(1) quantities per iteration; with
B <= 6 that is at most ~110 roundings of 1.1e-16 each, so 1e-13 relative per
array leaves an order of magnitude for cancellation (lduh subtracts
neighbouring fluxes, 1e-12 there)."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
from exahype_b200 import DeviceBuffer

pytestmark = pytest.mark.gpu
V = 5


def run(variant, dim, order, cells, q, dx, dt, pde):
    s = O.sizes(dim, order)
    k = E.BatchedADERDG(dim, order, dx, pde=pde)
    out = {n: DeviceBuffer(cells * s[n]) for n in ('lduh', 'qbnd', 'fbnd')}
    it = DeviceBuffer(cells, np.int32)
    E._lib.call('exa_tune_set', 3, variant)
    try:
        k.predictor_vi(cells, DeviceBuffer.from_array(q.ravel()), dt, out['lduh'], out['qbnd'], out['fbnd'], iters=it)
        return {n: b.download().reshape(cells, -1) for n, b in out.items()}, it.download()
    finally:
        E._lib.call('exa_tune_set', 3, 0)


@pytest.mark.parametrize('dim,order,cells,planar', [
    (2, 2, 1, 0), (2, 2, 13, 1), (2, 2, 29, 0), (2, 3, 7, 0), (2, 3, 17, 1), (2, 4, 4, 0), (2, 4, 11, 1),
    (2, 5, 1, 1), (2, 5, 4, 0), (2, 5, 11, 0), (3, 3, 1, 0), (3, 3, 5, 0), (3, 4, 1, 0), (3, 4, 5, 0), (3, 5, 3, 0)])
def test_pencil_vs_gather_and_oracle(dim, order, cells, planar):
    rng = np.random.default_rng(1000 * dim + 10 * order + cells)
    nn = (order + 1) ** dim
    q = np.zeros((cells, nn, V))
    # from nearly constant to rough, so the cells of a CTA stop at different iterations
    amp = 10.0 ** rng.uniform(-6, -0.6, (cells, 1))
    q[..., 0] = 1.0 + amp * rng.random((cells, nn))
    q[..., 1:4] = amp[..., None] * rng.standard_normal((cells, nn, 3))
    q[..., 4] = 2.5 + amp * rng.random((cells, nn))
    dx, dt = [0.05, 0.04, 0.03][:dim], 3e-4
    pde = E.PDE_EULER_PLANAR if planar else E.PDE_EULER
    a, ia = run(0, dim, order, cells, q, dx, dt, pde)
    b, ib = run(1, dim, order, cells, q, dx, dt, pde)
    assert np.array_equal(ia, ib)
    if cells > 3:
        assert len(set(ia)) > 1
    for c in range(cells):
        r = O.stp(dim, order, q[c].ravel(), dx, dt, planar=planar)
        assert ia[c] == r['iters']
        lduh = np.zeros(nn * V)
        O.lib().orc_volume_integral(dim, order, V, 1, lduh, r['lFhi'], np.array(dx))
        for n, ref in (('lduh', lduh), ('qbnd', r['lQhbnd']), ('fbnd', r['lFhbnd'])):
            tol = (1e-12 if n == 'lduh' else 1e-13) * np.abs(r['lFhi'] if n == 'lduh' else ref).max() / (
                min(dx) if n == 'lduh' else 1.0)
            assert np.abs(a[n][c] - ref).max() <= tol, (n, c)
            assert np.abs(a[n][c] - b[n][c]).max() <= tol, (n, c)


@pytest.mark.parametrize('dim,order,cells', [(2, 2, 29), (2, 3, 17), (2, 4, 11), (2, 5, 8), (3, 3, 5), (3, 4, 4),
                                             (3, 5, 3)])
def test_cells_of_nan(dim, order, cells):
    """Cells of nothing but NaN, cells with one NaN, and the cells beside them:
    the iteration limit and NaN for the first two, what they are alone for the
    others."""
    rng = np.random.default_rng(dim + order)
    nn = (order + 1) ** dim
    q = np.zeros((cells, nn, V))
    q[..., 0] = 1.0 + 0.1 * rng.random((cells, nn))
    q[..., 1:4] = 0.1 * rng.standard_normal((cells, nn, 3))
    q[..., 4] = 2.5 + 0.1 * rng.random((cells, nn))
    dx, dt = [0.05, 0.04, 0.03][:dim], 3e-4
    good, ig = run(0, dim, order, cells, q, dx, dt, E.PDE_EULER)
    q[0] = np.nan
    q[2, nn // 2, 1] = np.nan
    a, ia = run(0, dim, order, cells, q, dx, dt, E.PDE_EULER)
    for c in range(cells):
        if c in (0, 2):
            assert ia[c] == 2 * (order + 1)
            assert all(np.isnan(a[n][c]).all() for n in a)
        else:
            assert ia[c] == ig[c]
            assert all(np.array_equal(a[n][c], good[n][c]) for n in a)


@pytest.mark.parametrize('order,cells', [(2, 1), (2, 29), (2, 1184), (2, 1185), (5, 1), (5, 11), (5, 592), (5, 593)])
def test_few_2d_cells(order, cells):
    """Orders 2 and 5 take the line-owner form for few 2D cells (8 and 4 per SM;
    the sizes are those of 148 SMs): default, pencil (key 3 = 4) and line-owner
    (key 3 = 2) agree to the roundings above, with NaN cells among the others."""
    rng = np.random.default_rng(cells + order)
    nn = (order + 1) ** 2
    q = np.zeros((cells, nn, V))
    q[..., 0] = 1.0 + 0.1 * rng.random((cells, nn))
    q[..., 1:4] = 0.1 * rng.standard_normal((cells, nn, 3))
    q[..., 4] = 2.5 + 0.1 * rng.random((cells, nn))
    if cells > 10:
        q[3] = np.nan
        q[7, nn // 2, 1] = np.nan
    dx, dt = [0.05, 0.04], 3e-4
    a, ia = run(0, 2, order, cells, q, dx, dt, E.PDE_EULER)
    for variant in (2, 4):
        b, ib = run(variant, 2, order, cells, q, dx, dt, E.PDE_EULER)
        assert np.array_equal(ia, ib)
        for n in a:
            assert np.array_equal(np.isnan(a[n]), np.isnan(b[n]))
            # lduh is a difference of fluxes (about 3) over dx
            scale = 3.0 / min(dx) if n == 'lduh' else np.nanmax(np.abs(a[n]))
            assert np.nanmax(np.abs(a[n] - b[n])) <= (1e-12 if n == 'lduh' else 1e-13) * scale
