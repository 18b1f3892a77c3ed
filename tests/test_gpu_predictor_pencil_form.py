"""The pencil predictor itself (tuning key 3 = 4) at the few 2D cells of orders 2
and 5 for which the default is the line-owner form: 14 cells in 126 threads, 5
in 180, cells that straddle warps, partly filled blocks, blocks whose cells stop
at different iterations or hold NaN; against node-gather and the oracle, with
the tolerances of the tests it repeats.  And whole grids with the default and
with the pencil form, step by step against the oracle."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
import test_gpu_predictor_pencil as P

pytestmark = pytest.mark.gpu
TOL = 1e-12  # relative L2 per step, as for the other forms


@pytest.fixture
def pencil(monkeypatch):
    run = P.run
    monkeypatch.setattr(P, 'run', lambda variant, *a: run(variant or 4, *a))


@pytest.mark.parametrize('order,cells', [(2, 1), (2, 13), (2, 14), (2, 29), (5, 1), (5, 4), (5, 5), (5, 11), (5, 33)])
@pytest.mark.parametrize('planar', [0, 1])
def test_pencil_vs_gather_and_oracle(pencil, order, cells, planar):
    P.test_pencil_vs_gather_and_oracle(2, order, cells, planar)


@pytest.mark.parametrize('order,cells', [(2, 29), (2, 9), (5, 8), (5, 11)])
def test_cells_of_nan(pencil, order, cells):
    P.test_cells_of_nan(2, order, cells)


@pytest.mark.parametrize('variant', [0, 4])
@pytest.mark.parametrize('dim,order,n,planar', [(2, 2, (9, 7), 1), (2, 3, (9, 7), 0), (2, 4, (6, 7), 1), (2, 5, (6, 5), 0),
                                                (2, 5, (5, 6), 1), (3, 2, (3, 4, 3), 0), (3, 3, (3, 4, 3), 0),
                                                (3, 4, (3, 2, 3), 0), (3, 5, (2, 3, 2), 0)])
def test_grid_steps_vs_oracle(variant, dim, order, n, planar):
    E._lib.call('exa_tune_set', 3, variant)
    try:
        g = E.ADERDGGrid(dim, order, n, pde=E.PDE_EULER_PLANAR if planar else E.PDE_EULER)
        g.init(kind=0, param=5.0, seed=8, noise=1e-3)
        u = g.get_state()
        for s in range(4):
            dt = g.step(1, want_dt=True)[0]
            ref, _ = O.grid_step(dim, order, n, u, planar=planar)
            assert abs(dt - ref) <= 1e-13 * ref
            got = g.get_state()
            assert np.linalg.norm(got - u) <= TOL * np.linalg.norm(u), s
            u = got.copy()
        g.destroy()
    finally:
        E._lib.call('exa_tune_set', 3, 0)
