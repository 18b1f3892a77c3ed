"""2D orders 2 and 5 take the line-owner predictor for few cells (tuning key 3 =
2) and the pencil predictor for many (key 3 = 4): a cell's outputs and iteration
count are the same bits in both, so that they do not depend on how many cells
share a call.  Every output is compared exactly; NaN cells by where the NaN
are."""
import numpy as np
import pytest

import exahype_b200 as E
from test_gpu_predictor_place import V, around, predict, rough_cells, threshold_scales

pytestmark = pytest.mark.gpu


def same(a, b):
    assert np.array_equal(a[1], b[1])
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize('order', [2, 5])
@pytest.mark.parametrize('planar', [0, 1])
@pytest.mark.parametrize('cells', [1, 14, 29, 600, 1300])
def test_forms_agree(order, planar, cells):
    rng = np.random.default_rng(100 * order + cells)
    nn = (order + 1) ** 2
    amp = 10.0 ** rng.uniform(-8, -0.6, (cells, 1))  # the cells stop at different iterations
    q = np.zeros((cells, nn, V))
    q[..., 0] = 1.0 + amp * rng.random((cells, nn))
    q[..., 1:4] = amp[..., None] * rng.standard_normal((cells, nn, 3))
    q[..., 4] = 2.5 + amp * rng.random((cells, nn))
    if cells > 10:
        q[3] = np.nan
        q[7, nn // 2, 1] = np.nan
        q[9, 0, 0] = np.inf
        assert len(set(predict(2, order, q)[1])) > 2
    pde = E.PDE_EULER_PLANAR if planar else E.PDE_EULER
    line, pencil, default = (predict(v, order, q, pde) for v in (2, 4, 0))
    same(line, pencil)
    same(line, default)


@pytest.mark.parametrize('order', [2, 5])
def test_forms_stop_alike(order):
    """residuals within a few units in the last place of the tolerance"""
    q = rough_cells(order, 200, 31 + order)
    s = threshold_scales(2, order, q)
    for ulps in range(-6, 7):
        u = around(s, ulps)[:, None, None] * q
        same(predict(2, order, u), predict(4, order, u))
