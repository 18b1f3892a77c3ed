"""Batched 2D finite-volume updates on both sides of the counts where their
launch changes (row blocks of the Godunov sweep; threads per MUSCL-Hancock
patch: one and two patches per SM): a patch's new state, its ghost ring and its
admissible dt are the same bits whatever the batch, and those of the oracle to
1e-13 relative (four face terms of O(1) per cell)."""
import numpy as np
import pytest

import _oracle as O
import exahype_b200 as E
from exahype_b200 import DeviceBuffer, FVPatches

pytestmark = pytest.mark.gpu
V = 5


@pytest.mark.parametrize('scheme', [0, 1])
@pytest.mark.parametrize('P,npar,planar', [(3, 0, 0), (9, 2, 1), (10, 0, 0), (12, 1, 0), (14, 0, 1), (15, 0, 0),
                                           (16, 2, 0), (16, 0, 1), (31, 0, 0)])
def test_patch_same_in_any_batch(scheme, P, npar, planar):
    g, kinds = scheme + 1, 7
    S, D = P + 2 * g, V + npar
    rng = np.random.default_rng(P + 100 * scheme)
    q = np.zeros((kinds, S, S, D))
    q[..., 0] = 1.0 + 0.3 * rng.random((kinds, S, S))
    q[..., 1:4] = 0.3 * rng.standard_normal((kinds, S, S, 3))
    q[..., 4] = 2.5 + rng.random((kinds, S, S)) + 0.5 * (q[..., 1:4] ** 2).sum(-1) / q[..., 0]
    q[..., V:] = rng.random((kinds, S, S, npar))
    dx, dt = [0.5, 0.7], 0.1 * 0.5 / P
    k = FVPatches(P, g, dx, pde=E.PDE_EULER_PLANAR if planar else E.PDE_EULER, npar=npar)
    update = k.godunov_update if scheme == 0 else k.musclhancock_update
    f = O.lib().orc_fv_godunov_2d if scheme == 0 else O.lib().orc_fv_musclhancock_2d
    first = None
    for n in (kinds, 148, 149, 296, 297, 700):
        which = np.arange(n) % kinds
        old, new = DeviceBuffer.from_array(q[which].ravel()), DeviceBuffer.from_array(q[which].ravel())
        adm = DeviceBuffer(n)
        update(n, new, old, dt, adm)
        got, dts = new.download().reshape(n, -1), adm.download()
        if first is None:
            first = got, dts
            for i in range(kinds):
                ref = q[i].ravel().copy()
                want = f(P, g, V, npar, planar, ref, q[i].ravel().copy(), np.array(dx), dt)
                assert np.abs(got[i] - ref).max() <= 1e-13 * np.abs(ref).max(), i
                assert abs(dts[i] - want) <= 1e-14 * want, i
        assert np.array_equal(got, first[0][which])
        assert np.array_equal(dts, first[1][which])
