"""Batched updates whose output is their input (patches of one strip of columns
and one block of rows, whatever their number): the same states as into another
array that holds the input."""
import numpy as np
import pytest

import exahype_b200 as E
from exahype_b200 import DeviceBuffer, FVPatches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scheme,P', [(0, 1), (0, 3), (0, 8), (0, 14), (0, 30), (1, 3), (1, 8), (1, 16)])
@pytest.mark.parametrize('n', [1, 50, 700])
def test_in_place(scheme, P, n):
    g = scheme + 1
    S = P + 2 * g
    rng = np.random.default_rng(P + n)
    q = np.zeros((n, S, S, 5))
    q[..., 0] = 1.0 + 0.3 * rng.random((n, S, S))
    q[..., 1:4] = 0.3 * rng.standard_normal((n, S, S, 3))
    q[..., 4] = 2.5 + rng.random((n, S, S))
    k = FVPatches(P, g, [0.5, 0.7])
    update = k.godunov_update if scheme == 0 else k.musclhancock_update
    old, new, both = (DeviceBuffer.from_array(q.ravel()) for _ in range(3))
    d0, d1 = DeviceBuffer(n), DeviceBuffer(n)
    for _ in range(5):
        new.upload(q.ravel())
        both.upload(q.ravel())
        update(n, new, old, 0.02 / P, d0)
        update(n, both, both, 0.02 / P, d1)
        assert np.array_equal(new.download(), both.download())
        assert np.array_equal(d0.download(), d1.download())
