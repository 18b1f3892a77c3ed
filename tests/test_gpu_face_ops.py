"""The batched cell-local and face operators on every order of the predictor
(Riemann on a face list, surface integral, update, stable dt) at counts that
leave the last warp or CTA partly empty, against the oracle.  Each result is
a sum of at most 2 DIM (surface) or B^(DIM-1) (face average) products: 1e-13
relative covers their reordering with two orders of magnitude to spare."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
from exahype_b200 import DeviceBuffer

pytestmark = pytest.mark.gpu
V = 5


@pytest.mark.parametrize('dim', [2, 3])
@pytest.mark.parametrize('order', [2, 3, 4, 5])
@pytest.mark.parametrize('cells', [1, 2, 13])
def test_face_ops_vs_oracle(dim, order, cells):
    rng = np.random.default_rng(100 * dim + 10 * order + cells)
    B = order + 1
    nn, nf = B ** dim, B ** (dim - 1)
    dx = [0.1, 0.07, 0.05][:dim]
    k = E.BatchedADERDG(dim, order, dx)

    def states(*shape):
        q = np.zeros(shape + (V,))
        q[..., 0] = 1.0 + 0.2 * rng.random(shape)
        q[..., 1:4] = 0.3 * rng.standard_normal(shape + (3,))
        q[..., 4] = 2.5 + 0.3 * rng.random(shape)
        return q

    q, qb = states(cells, nn), states(cells, 2 * dim, nf)
    lduh = rng.standard_normal((cells, nn * V))
    fb = rng.standard_normal((cells, 2 * dim, nf * V))
    d_luh, d_lduh = DeviceBuffer.from_array(q.ravel()), DeviceBuffer.from_array(lduh)
    d_qb, d_fb, dt_cell = DeviceBuffer.from_array(qb.ravel()), DeviceBuffer.from_array(fb.ravel()), DeviceBuffer(cells)

    # every direction of every cell against its right neighbour in the list
    left = np.repeat(np.arange(cells, dtype=np.int32), dim)
    right = ((left + 1) % cells).astype(np.int32)
    dirs = np.tile(np.arange(dim, dtype=np.int32), cells)
    k.riemann_faces(left.size, *[DeviceBuffer.from_array(a) for a in (left, right, dirs)], d_qb, d_fb)
    want = fb.copy()
    for l, r, d in zip(left, right, dirs):
        fl, fr = want[l, 2 * d + 1].copy(), want[r, 2 * d].copy()
        O.lib().orc_riemann(dim, order, V, 0, 0, fl, fr, qb[l, 2 * d + 1].ravel().copy(), qb[r, 2 * d].ravel().copy(), d)
        want[l, 2 * d + 1], want[r, 2 * d] = fl, fr
    got = d_fb.download().reshape(fb.shape)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()

    k.surface_integral(cells, d_lduh, d_fb)
    k.stable_dt(cells, d_luh, dt_cell)
    dts = dt_cell.download()
    k.solution_update(cells, d_luh, d_lduh, 3e-3)
    got_l, got_u = d_lduh.download().reshape(cells, -1), d_luh.download().reshape(cells, -1)
    for c in range(cells):
        ref = lduh[c].copy()
        O.lib().orc_surface_integral(dim, order, V, ref, got[c].ravel().copy(), np.array(dx))
        assert np.abs(got_l[c] - ref).max() <= 1e-13 * np.abs(ref).max()
        want_dt = O.lib().orc_stable_dt(dim, order, V, 0, 0, q[c].ravel().copy(), np.array(dx), 0.9)
        assert abs(dts[c] - want_dt) <= 1e-14 * want_dt
        ref = q[c].ravel().copy()
        O.lib().orc_solution_update(dim, order, V, 0, ref, got_l[c].copy(), 3e-3)
        assert np.abs(got_u[c] - ref).max() <= 1e-13 * np.abs(ref).max()
