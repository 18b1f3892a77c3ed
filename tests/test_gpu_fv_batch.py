"""Batched 2D finite-volume updates (exa_fv_godunov_update,
exa_fv_musclhancock_update) at the edges of their kernels' packing: patches
of 1 cell to more than one strip (30 columns) or row block (32 rows), several
patches side by side in a warp with a partial last warp, thick ghost layers,
parameters, uneven cell sizes.  Against the oracle: the whole luh_new, the
first ghost layer that the boundary faces reach included, and the admissible
dt per patch, which is also NULL-able.  A cell sums four face terms of O(1):
1e-13 relative is the bar of the other finite-volume parity tests."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
from exahype_b200 import DeviceBuffer, FVPatches

pytestmark = pytest.mark.gpu
V = 5


@pytest.mark.parametrize('scheme', [0, 1])
@pytest.mark.parametrize('P,extra,n,npar,planar', [
    (1, 0, 25, 0, 0), (2, 0, 9, 0, 1), (5, 1, 11, 2, 0), (9, 0, 5, 0, 0), (10, 0, 33, 0, 0), (14, 0, 3, 1, 0),
    (15, 2, 2, 0, 0), (16, 0, 2, 0, 1), (17, 0, 2, 0, 0), (29, 0, 2, 0, 0), (30, 0, 1, 0, 0), (31, 0, 2, 0, 0),
    (33, 1, 2, 1, 0), (64, 0, 2, 0, 0)])
def test_batch_update_vs_oracle(scheme, P, extra, n, npar, planar):
    g = scheme + 1 + extra
    S, D = P + 2 * g, V + npar
    rng = np.random.default_rng(100 * P + 10 * scheme + n)
    q = np.zeros((n, S, S, D))
    q[..., 0] = 1.0 + 0.3 * rng.random((n, S, S))
    q[..., 1:4] = 0.3 * rng.standard_normal((n, S, S, 3))
    q[..., 4] = 2.5 + rng.random((n, S, S)) + 0.5 * (q[..., 1:4] ** 2).sum(-1) / q[..., 0]
    q[..., V:] = rng.random((n, S, S, npar))
    dx = [0.5, 0.7]
    dt = 0.1 * 0.5 / P
    k = FVPatches(P, g, dx, pde=E.PDE_EULER_PLANAR if planar else E.PDE_EULER, npar=npar)
    update = k.godunov_update if scheme == 0 else k.musclhancock_update
    old, new, adm = DeviceBuffer.from_array(q.ravel()), DeviceBuffer.from_array(q.ravel()), DeviceBuffer(n)
    update(n, new, old, dt, adm)
    got, dts = new.download().reshape(n, -1), adm.download()
    new.upload(q.ravel())
    update(n, new, old, dt)
    assert np.array_equal(new.download().reshape(n, -1), got)
    assert np.array_equal(old.download(), q.ravel())
    f = O.lib().orc_fv_godunov_2d if scheme == 0 else O.lib().orc_fv_musclhancock_2d
    for i in range(n):
        ref = q[i].ravel().copy()
        want = f(P, g, V, npar, planar, ref, q[i].ravel().copy(), np.array(dx), dt)
        assert np.abs(got[i] - ref).max() <= 1e-13 * np.abs(ref).max(), i
        assert abs(dts[i] - want) <= 1e-14 * want, i
