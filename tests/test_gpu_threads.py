"""Host threads that call the same kernel with different shared-memory needs at
once (the entry points are reentrant): the size a function may be launched with
is one value per device, and a call of a small size must not lower it under
another thread's feet."""
import ctypes as C
import threading

import numpy as np
import pytest

import exahype_b200 as E
from exahype_b200 import DeviceBuffer, limiter
from exahype_b200.fv import FVPatches

pytestmark = pytest.mark.gpu
V = 5


def hammer(jobs, calls):
    """every job in a thread of its own, `calls` times; the errors they raised"""
    errors, start = [], threading.Barrier(len(jobs))

    def work(job):
        try:
            E.lib().exa_set_device(0)
            start.wait()
            for _ in range(calls):
                job()
        except Exception as e:  # reported by the caller
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    E._lib.call('exa_stream_synchronize', None)
    return errors


def gas(points, seed):
    q = np.zeros((points, V))
    rng = np.random.default_rng(seed)
    q[:, 0] = 1.0 + 0.1 * rng.random(points)
    q[:, 4] = 2.5 + 0.1 * rng.random(points)
    return q.ravel()


def test_musclhancock_batches_of_two_sizes():
    jobs, keep = [], []
    for patch in (16, 3, 16, 5):
        f = FVPatches(patch, 2, [0.1, 0.1])
        q = DeviceBuffer.from_array(gas(f.cells_per_patch, patch))
        out = DeviceBuffer.from_array(gas(f.cells_per_patch, patch))
        keep += [f, q, out]
        jobs.append(lambda f=f, q=q, out=out: f.musclhancock_update(1, out, q, 1e-9))
    assert hammer(jobs, 3000) == []


@pytest.mark.parametrize('dim,order', [(3, 3), (2, 4)])
def test_projections_of_two_sizes(dim, order):
    jobs, keep = [], []
    for ghost, cells in ((2, 1), (0, 1), (2, 40), (0, 3000)):
        luh = DeviceBuffer.from_array(gas(cells * (order + 1) ** dim, ghost))
        lim = DeviceBuffer(cells * limiter.patch_doubles(dim, order, ghost=ghost))
        lim.zero()
        keep += [luh, lim]
        jobs.append(lambda g=ghost, n=cells, a=luh, b=lim: limiter.project_on_fv(dim, order, n, a, b, ghost=g))
        out = DeviceBuffer(cells * (order + 1) ** dim * V)
        keep.append(out)
        jobs.append(lambda g=ghost, n=cells, a=lim, b=out: limiter.project_on_dg(dim, order, n, a, b, ghost=g))
    assert hammer(jobs, 1500) == []


def test_3d_patches_of_two_sizes():
    jobs, keep = [], []
    for patch in (10, 2, 8, 3):
        f = FVPatches(patch, 2, [0.1, 0.1, 0.1], dim=3)
        q = DeviceBuffer.from_array(gas(f.cells_per_patch, patch))
        out = DeviceBuffer.from_array(gas(f.cells_per_patch, patch))
        keep += [f, q, out]
        jobs.append(lambda f=f, q=q, out=out: f.musclhancock_update(1, out, q, 1e-9))
    assert hammer(jobs, 1500) == []


def test_limited_grids_of_two_orders():
    """the subcell patches of two grids, stepped by two threads"""
    grids = []
    for order in (2, 5):
        g = E.ADERDGGrid(2, order, (6, 5))
        g.init(kind=0, param=5.0, seed=order, noise=1e-3)
        g.set_limiter()
        grids.append(g)
    assert hammer([lambda g=g: g.step(1) for g in grids], 300) == []
    for g in grids:
        g.destroy()
