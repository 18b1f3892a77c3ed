"""Performance cases: what users of this library run, through its public Python entry points.

Kinds of work (the "kind" of a case):

* grid       ADERDGGrid.step: one uniform grid, 2D or 3D, orders 2..5, FP64 or mixed precision,
             periodic or with outflow / reflecting walls, replayed as a CUDA graph;
* traversal  BatchedADERDG: the device entry points that a host code with its own mesh calls once per
             traversal (predictor, Riemann solves on a face list, surface integral, update, stable dt);
* ensemble   Ensemble.step: many independent 2D solves of uneven size and order;
* serving    Server.tick: resident 2D ADER-DG and finite-volume requests advanced together;
* fv         FVGrid.step: one periodic 2D finite-volume patch, Godunov or MUSCL-Hancock;
* patches    FVPatches: batches of small 2D / 3D finite-volume patches with ghost layers;
* limiting   ADERDGGrid.step with the a-posteriori subcell limiter;
* limiter    the limiter's batched kernels (DMP check, projections) on device-resident cells.

exact() restates each of these in plain FP64 torch from the schemes' definitions.
"""
import ctypes
import math

import numpy as np
import torch

import exahype_b200 as E
from exahype_b200 import limiter
from exahype_b200 import serving as S
from exahype_b200.fv import FVGrid, FVPatches

GAMMA = 1.4
CFL = 0.9
PNPM = (1.0, 0.33, 0.17, 0.1, 0.069, 0.045)
PERIODIC, OUTFLOW, REFLECT = 0, 1, 2


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest call a user makes: the 2D N=3 27x27 sine-wave run, one step per call.
        dict(name='grid2d_n3_27', kind='grid', dim=2, order=3, nx=27, ny=27, nz=1, mixed=False, bcx=0, bcy=0, bcz=0),
        # A ragged 2D domain between walls, the highest order.
        dict(name='grid2d_n5_walls', kind='grid', dim=2, order=5, nx=211, ny=131, nz=1, mixed=False,
             bcx=OUTFLOW, bcy=REFLECT, bcz=0),
        # The benchmark workload: 3D Euler N=4 on 81^3 cells, FP64 and mixed precision.
        dict(name='grid3d_n4_81', kind='grid', dim=3, order=4, nx=81, ny=81, nz=81, mixed=False, bcx=0, bcy=0, bcz=0),
        dict(name='grid3d_n4_81_mixed', kind='grid', dim=3, order=4, nx=81, ny=81, nz=81, mixed=True,
             bcx=0, bcy=0, bcz=0),
        # A 3D production run at the next lower order on an uneven box with walls.
        dict(name='grid3d_n3_walls', kind='grid', dim=3, order=3, nx=53, ny=37, nz=41, mixed=False,
             bcx=REFLECT, bcy=OUTFLOW, bcz=PERIODIC),
        # A host code with its own mesh: one traversal's kernels over a face list.
        dict(name='traversal3d_n4', kind='traversal', dim=3, order=4, nx=31, ny=31, nz=31),
        # 512 independent 2D solves (orders 2..5, sides 9..81), five steps per call.
        dict(name='ensemble_512', kind='ensemble', solves=512, lo=9, hi=81, mix=2024, mixed=False, steps=5),
        # One tick of the serving engine with a resident mix of requests.
        dict(name='serving_24', kind='serving', dg=6, fv=18, mix=2524),
        # One periodic MUSCL-Hancock patch, larger than the L2 cache.
        dict(name='fv_muscl_4096', kind='fv', scheme=1, patch=4096),
        # The finite-volume demonstrator's layout: many 2D patches of 10x10 cells.
        dict(name='patches2d_godunov_10', kind='patches', dim=2, scheme=0, patch=10, count=40000),
        # An explosion stabilised by the subcell limiter.
        dict(name='limiting2d_n3_243', kind='limiting', dim=2, order=3, n=243),
        # The limiter's kernels on a batch of 3D N=4 cells.
        dict(name='limiter3d_n4', kind='limiter', dim=3, order=4, count=40000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['grid', 'grid', 'grid', 'traversal', 'ensemble', 'serving', 'fv', 'patches', 'limiting',
                       'limiter'])
    if kind in ('grid', 'traversal'):
        dim = rng.choice([2, 3])
        order = rng.randint(2, 5)
        # cells per direction up to about 2^22 nodes (2D) / 2^25 nodes (3D)
        top = (2 ** 22 if dim == 2 else 2 ** 25) ** (1.0 / dim) / (order + 1)
        if kind == 'traversal':
            top *= 0.5
        side = [_log_int(rng, 5, top) if i == 0 else 0 for i in range(3)]
        side[1] = max(3, int(side[0] * rng.uniform(0.6, 1.0)))
        side[2] = max(3, int(side[0] * rng.uniform(0.6, 1.0))) if dim == 3 else 1
        c = dict(kind=kind, dim=dim, order=order, nx=side[0], ny=side[1], nz=side[2])
        if kind == 'grid':
            walls = rng.random() < 0.3
            c.update(mixed=rng.random() < 0.35, bcx=rng.randint(0, 2) if walls else 0,
                     bcy=rng.randint(0, 2) if walls else 0, bcz=rng.randint(0, 2) if walls and dim == 3 else 0)
        return c
    if kind == 'ensemble':
        lo = rng.randint(9, 30)
        return dict(kind=kind, solves=_log_int(rng, 8, 256), lo=lo, hi=lo + rng.randint(5, 50),
                    mix=rng.randint(1, 1 << 30), mixed=rng.random() < 0.5, steps=rng.randint(1, 5))
    if kind == 'serving':
        return dict(kind=kind, dg=rng.randint(1, 10), fv=rng.randint(2, 24), mix=rng.randint(1, 1 << 30))
    if kind == 'fv':
        return dict(kind=kind, scheme=rng.randint(0, 1), patch=_log_int(rng, 64, 4200))
    if kind == 'patches':
        dim = rng.choice([2, 3])
        scheme = rng.randint(0, 1)
        patch = _log_int(rng, 5, 64) if dim == 2 else rng.randint(5, 11)
        count = _log_int(rng, 50, 4.0e6 / patch ** dim)
        return dict(kind=kind, dim=dim, scheme=scheme, patch=patch, count=min(count, 60000))
    if kind == 'limiting':
        dim = rng.choice([2, 2, 3])
        order = rng.randint(2, 4)
        return dict(kind=kind, dim=dim, order=order, n=_log_int(rng, 40, 300) if dim == 2 else rng.randint(12, 30))
    dim = rng.choice([2, 3])
    order = rng.randint(2, 5)
    return dict(kind='limiter', dim=dim, order=order, count=_log_int(rng, 300, 6.0e6 / (order + 1) ** dim))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(int(seed))


def _uniform(seed, shape, lo, hi):
    return torch.rand(shape, generator=_gen(seed), device='cuda', dtype=torch.float64) * (hi - lo) + lo


class _DeviceMemory:
    """Memory of the library seen by torch without a copy."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = dict(shape=(int(n),), typestr='<f8', data=(int(ptr), False), version=3)


def _view(owner, ptr, n):
    """Tensor over n doubles at ptr, device memory of `owner`, which lives as long as the tensor does."""
    t = torch.as_tensor(_DeviceMemory(getattr(ptr, 'value', ptr), n), device='cuda')
    t.owner = owner
    return t


class _Buffer:
    """A torch tensor in the place of a device buffer: the entry points take its .ptr."""

    def __init__(self, t):
        self.t = t
        self.ptr = ctypes.c_void_p(t.data_ptr())


def _cells(c):
    return [c['nx'], c['ny']] + ([c['nz']] if c['dim'] == 3 else [])


def _lengths(c):
    n = _cells(c)
    return [k / n[0] for k in n]  # cubic cells, unit length in x


def _nodes(order):
    x, w = np.polynomial.legendre.leggauss(order + 1)
    return (x + 1) / 2, w / 2


def _node_coordinates(dim, order, n, length):
    """x, y (and z) of every node, each broadcastable to [nz, ny, nx, B, B, B] ([ny, nx, B, B] in 2D)."""
    xi = torch.as_tensor(_nodes(order)[0], device='cuda')
    out = []
    for d in range(dim):
        t = (torch.arange(n[d], device='cuda', dtype=torch.float64)[:, None] + xi[None, :]) * (length[d] / n[d])
        shape = [1] * (2 * dim)
        shape[dim - 1 - d] = n[d]
        shape[2 * dim - 1 - d] = order + 1
        out.append(t.reshape(shape))
    return out


def _conserved(rho, u, v, p):
    q = torch.zeros(rho.shape + (5,), device='cuda', dtype=torch.float64)
    q[..., 0] = rho
    q[..., 1] = rho * u
    q[..., 2] = rho * v
    q[..., 4] = p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)
    return q


def _dg_state(case, seed):
    """Nodal state [cells, nodes, 5]: the isentropic vortex in 3D and the density wave in 2D, or a pressure pulse at
    rest between walls, with seeded density noise of amplitude 1e-3."""
    dim, order, n, length = case['dim'], case['order'], _cells(case), _lengths(case)
    x = _node_coordinates(dim, order, n, length)
    shape = torch.broadcast_shapes(*[t.shape for t in x])
    r = [t / length[d] - 0.5 for d, t in enumerate(x)]
    if case.get('bcx', 0) or case.get('bcy', 0) or case.get('bcz', 0):
        p = 1.0 + 0.2 * torch.exp(-20.0 * sum(t * t for t in r))
        rho, u, v = p ** (1 / GAMMA), torch.zeros(shape, device='cuda', dtype=torch.float64), 0.0
        rho = rho.expand(shape)
    elif dim == 3:
        xb, yb, eps = r[0] / 0.1, r[1] / 0.1, 5.0
        e = torch.exp(0.5 * (1.0 - xb * xb - yb * yb))
        u = (1.0 - eps / (2 * math.pi) * yb * e).expand(shape)
        v = (1.0 + eps / (2 * math.pi) * xb * e).expand(shape)
        t = 1.0 - (GAMMA - 1) * eps * eps / (8 * GAMMA * math.pi ** 2) * e * e
        rho = (t ** (1 / (GAMMA - 1))).expand(shape)
        p = rho * t
    else:
        rho = (1.0 + 0.2 * torch.sin(2 * math.pi * (r[0] + r[1]))).expand(shape)
        u, v, p = torch.ones(shape, device='cuda', dtype=torch.float64), 1.0, 1.0
    rho = rho * (1.0 + 1e-3 * _uniform(seed, shape, -1.0, 1.0))
    return _conserved(rho, u, v, p).reshape(-1, (order + 1) ** dim, 5)


def _explosion(case, seed):
    """Density 1 / pressure 1 inside a circle (sphere), 0.125 / 0.1 outside, at rest; centre and radius from the seed."""
    dim, order, n = case['dim'], case['order'], case['n']
    rng = np.random.default_rng(seed)
    centre, radius = rng.uniform(0.45, 0.55, dim), rng.uniform(0.2, 0.28)
    x = _node_coordinates(dim, order, [n] * dim, [1.0] * dim)
    inside = sum((x[d] - centre[d]) ** 2 for d in range(dim)) < radius ** 2
    one = torch.ones(inside.shape, device='cuda', dtype=torch.float64)
    q = _conserved(torch.where(inside, one, 0.125 * one), 0.0 * one, 0.0, torch.where(inside, one, 0.1 * one))
    return q.reshape(-1, (order + 1) ** dim, 5)


def _fv_state(dim, patch, ghost, count, seed, domain):
    """[count, S.., 5] padded patches: one periodic density wave over the domain (domain=True: the patch is the domain
    and its ghosts the periodic images), or patches cut from a smooth field with noise."""
    side = patch + 2 * ghost
    noise = 1e-3 * _uniform(seed, (count,) + (patch if domain else side,) * dim, -1.0, 1.0)
    k = (torch.arange(noise.shape[1], device='cuda', dtype=torch.float64) + 0.5) / patch
    axes = [k.reshape([-1 if a == d else 1 for a in range(dim)]) for d in range(dim)]
    phase = torch.zeros((count,) + (1,) * dim, device='cuda', dtype=torch.float64)
    if not domain:
        phase = _uniform(seed + 1, phase.shape, 0.0, 1.0)
    scale = 1.0 if domain else 0.1
    wave = torch.sin(2 * math.pi * (scale * sum(axes)[None] + phase))
    rho = (1.0 + 0.2 * wave) * (1.0 + noise)
    u, v = 1.0 + 0.1 * wave, 0.7 - 0.1 * wave
    p = 1.0 + 0.05 * wave
    q = _conserved(rho, u.expand(rho.shape), v.expand(rho.shape), p.expand(rho.shape))
    if domain:
        for a in range(dim):
            q = torch.cat([q.narrow(1 + a, patch - ghost, ghost), q, q.narrow(1 + a, 0, ghost)], 1 + a)
    return q.contiguous()


def _mix(case):
    """Sizes of an ensemble's solves / a server's requests (the case's own mix)."""
    rng = np.random.default_rng(case['mix'])
    if case['kind'] == 'ensemble':
        return [(int(rng.integers(2, 6)), int(rng.integers(case['lo'], case['hi'] + 1)))
                for _ in range(case['solves'])]
    dg = [(int(rng.integers(2, 6)), int(round(math.exp(rng.uniform(math.log(9), math.log(243))))))
          for _ in range(case['dg'])]
    fv = [int(round(math.exp(rng.uniform(math.log(64), math.log(1024))))) for _ in range(case['fv'])]
    return dg, fv


def _amplitudes(count, seed):
    return [float(a) for a in np.random.default_rng(seed).uniform(0.05, 0.3, count)]


def _faces(case):
    """Face list of a periodic mesh: left and right cell and the normal direction of every face, and the cells'
    neighbours [cells, 2 dim]."""
    dim, n = case['dim'], _cells(case)
    idx = torch.arange(math.prod(n), device='cuda').reshape(n[::-1])
    nb = []
    for d in range(dim):
        nb += [torch.roll(idx, 1, dim - 1 - d).reshape(-1), torch.roll(idx, -1, dim - 1 - d).reshape(-1)]
    left = torch.cat([idx.reshape(-1)] * dim)
    right = torch.cat([nb[2 * d + 1] for d in range(dim)])
    direction = torch.arange(dim, device='cuda').repeat_interleave(idx.numel())
    return left.int(), right.int(), direction.int(), torch.stack(nb, 1)


def _dt_factor(order):
    return CFL * PNPM[order]


# ------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    return _PREPARE[case['kind']](case, seed)


def run(state):
    return _RUN[state['kind']](state)


def _prepare_grid(case, seed):
    g = E.ADERDGGrid(case['dim'], case['order'], _cells(case), _lengths(case),
                     precision=E.PREC_MIXED if case['mixed'] else E.PREC_FP64)
    bc = [case['bcx'], case['bcy'], case['bcz']][:case['dim']]
    if any(bc):
        g.set_boundary(bc)
    g.set_state(_dg_state(case, seed).reshape(-1).cpu().numpy())
    g.use_graph(True)
    return dict(kind='grid', grid=g, state=_view(g, g.device_state_ptr(), g.state_size))


def _run_grid(s):
    s['grid'].step(1)
    return s['state']


def _prepare_limiting(case, seed):
    g = E.ADERDGGrid(case['dim'], case['order'], [case['n']] * case['dim'])
    g.set_state(_explosion(case, seed).reshape(-1).cpu().numpy())
    g.set_limiter()
    g.use_graph(True)
    return dict(kind='limiting', grid=g, state=_view(g, g.device_state_ptr(), g.state_size))


def _prepare_traversal(case, seed):
    dim, order, n = case['dim'], case['order'], _cells(case)
    u = _dg_state(case, seed)
    left, right, direction, _ = _faces(case)
    dx = [1.0 / n[0]] * dim
    dt = 0.7 * float(_cell_dt(u, dim, order, torch.tensor([dx], device='cuda', dtype=torch.float64)).min())
    cells = u.shape[0]
    face = cells * 2 * dim * (order + 1) ** (dim - 1) * 5

    def buf(count):
        return _Buffer(torch.zeros(count, device='cuda', dtype=torch.float64))

    return dict(kind='traversal', k=E.BatchedADERDG(dim, order, dx), cells=cells, dt=dt, luh=_Buffer(u.reshape(-1)),
                lduh=buf(u.numel()), qb=buf(face), fb=buf(face), dt_cell=buf(cells), nfaces=left.numel(),
                left=_Buffer(left), right=_Buffer(right), direction=_Buffer(direction))


def _run_traversal(s):
    k = s['k']
    k.predictor_vi(s['cells'], s['luh'], s['dt'], s['lduh'], s['qb'], s['fb'])
    k.riemann_faces(s['nfaces'], s['left'], s['right'], s['direction'], s['qb'], s['fb'])
    k.surface_integral(s['cells'], s['lduh'], s['fb'])
    k.solution_update(s['cells'], s['luh'], s['lduh'], s['dt'])
    k.stable_dt(s['cells'], s['luh'], s['dt_cell'])
    return dict(luh=s['luh'].t, lduh=s['lduh'].t, fluxes=s['fb'].t, dt=s['dt_cell'].t)


def _prepare_ensemble(case, seed):
    mix = _mix(case)
    cfgs = [E.solve_config(o, (n, n), ic_kind=1, ic_param=a) for (o, n), a in zip(mix, _amplitudes(len(mix), seed))]
    arena = int(sum(E.ensemble.footprint(c) for c in cfgs) * 1.05) + (1 << 24)
    ens = E.Ensemble(len(cfgs), arena, precision=E.PREC_MIXED if case['mixed'] else E.PREC_FP64)
    slots = [ens.add(c) for c in cfgs]
    ens.set_launch_mode(1)
    ens.use_graph(True)
    views = [_view(ens, ens.device_state_ptr(k), ens.state_size(k)) for k in slots]
    ens.synchronize()
    return dict(kind='ensemble', ens=ens, steps=case['steps'], views=views)


def _run_ensemble(s):
    s['ens'].step(s['steps'])
    s['ens'].synchronize()
    states = torch.cat(s['views'])
    torch.cuda.current_stream().synchronize()  # the next step, on the ensemble's stream, overwrites what this reads
    return states


def _prepare_serving(case, seed):
    dg, fv = _mix(case)
    amps = _amplitudes(len(dg) + len(fv), seed)
    reqs = [S.dg_request(o, n, 10 ** 9, ic_param=a) for (o, n), a in zip(dg, amps)]
    reqs += [S.fv_request(n, 10 ** 9, ic_param=a) for n, a in zip(fv, amps[len(dg):])]
    srv = S.Server(int(sum(S.footprint(r) for r in reqs) * 1.05) + (1 << 24), max_requests=64)
    srv.tune(launch_mode=1, use_graph=True)
    ids = [srv.submit(r) for r in reqs]
    return dict(kind='serving', server=srv, ids=ids, sizes=[S.result_size(r) for r in reqs], views={})


def _run_serving(s):
    s['server'].tick()
    out = []
    for rid, size in zip(s['ids'], s['sizes']):
        p = s['server'].device_state_ptr(rid)
        if p not in s['views']:
            s['views'][p] = _view(s['server'], p, size)
        out.append(s['views'][p])
    return out


def _prepare_fv(case, seed):
    g = FVGrid(case['scheme'], case['patch'])
    g.set_state(_fv_state(2, case['patch'], g.ghost, 1, seed, True).reshape(-1).cpu().numpy())
    return dict(kind='fv', grid=g, views={})


def _run_fv(s):
    s['grid'].step(1)
    p = s['grid'].device_state_ptr().value
    if p not in s['views']:
        s['views'][p] = _view(s['grid'], p, s['grid'].state_size)
    return s['views'][p]


def _prepare_patches(case, seed):
    dim, patch, ghost = case['dim'], case['patch'], case['scheme'] + 1
    u = _fv_state(dim, patch, ghost, case['count'], seed, False)
    new = torch.empty_like(u)
    dt = torch.zeros(case['count'], device='cuda', dtype=torch.float64)
    k = FVPatches(patch, ghost, [1.0] * dim, dim=dim)
    return dict(kind='patches', count=case['count'], dt=0.05 / patch,
                update=k.godunov_update if case['scheme'] == 0 else k.musclhancock_update,
                luh=_Buffer(u), luh_new=_Buffer(new), max_dt=_Buffer(dt))


def _run_patches(s):
    s['luh_new'].t.copy_(s['luh'].t)  # the update advances a copy of the old state in place
    s['update'](s['count'], s['luh_new'], s['luh'], s['dt'], s['max_dt'])
    return s['luh_new'].t, s['max_dt'].t


def _prepare_limiter(case, seed):
    dim, order, count = case['dim'], case['order'], case['count']
    u = _uniform(seed, (count, (order + 1) ** dim, 5), 0.5, 2.0)
    lim = torch.zeros((count, limiter.patch_doubles(dim, order, ghost=1)), device='cuda', dtype=torch.float64)
    lo = _uniform(seed + 1, (count, 2 * dim, 5), 0.1, 0.5)
    hi = _uniform(seed + 2, (count, 2 * dim, 5), 2.0, 2.4)
    return dict(kind='limiter', dim=dim, order=order, count=count, luh=_Buffer(u), lim=_Buffer(lim),
                back=_Buffer(torch.zeros_like(u)), lo=_Buffer(lo), hi=_Buffer(hi),
                ok=_Buffer(torch.zeros(count, device='cuda', dtype=torch.int32)))


def _run_limiter(s):
    dim, order, count = s['dim'], s['order'], s['count']
    limiter.dmp(dim, order, count, s['luh'], s['lo'], s['hi'], s['ok'], 1e-4, 1e-3)
    limiter.project_on_fv(dim, order, count, s['luh'], s['lim'], ghost=1)
    limiter.project_on_dg(dim, order, count, s['lim'], s['back'], ghost=1)
    return s['ok'].t, s['lo'].t, s['hi'].t, s['lim'].t, s['back'].t


_PREPARE = dict(grid=_prepare_grid, traversal=_prepare_traversal, ensemble=_prepare_ensemble,
                serving=_prepare_serving, fv=_prepare_fv, patches=_prepare_patches, limiting=_prepare_limiting,
                limiter=_prepare_limiter)
_RUN = dict(grid=_run_grid, traversal=_run_traversal, ensemble=_run_ensemble, serving=_run_serving, fv=_run_fv,
            patches=_run_patches, limiting=_run_grid, limiter=_run_limiter)


# ------------------------------------------------------------------ work
def _dg_work(dim, order):
    """Bytes (state in and out) and floating-point operations of one ADER-DG cell-update: four Picard iterations
    (the first evaluates one time slice), outputs, face solves and update."""
    b, v = order + 1, 5
    nn = b ** dim
    flux, node = 10 * dim + 1, 2 * dim * b * v
    iteration = b * nn * (node + flux + 2 * b * v)
    post = nn * (flux + node + 4 * b * v + 2 * b * v * dim) + 2 * dim * b ** (dim - 1) * (6 * v + 16) + nn * 6 * dim * v
    return 16 * nn * v, (3 + 1.0 / b) * iteration + post


_FV_FLOPS = {(2, 0): 304, (2, 1): 558, (3, 0): 456, (3, 1): 840}


def work(case):
    kind = case['kind']
    if kind in ('grid', 'traversal', 'limiting'):
        dim, order = case['dim'], case['order']
        cells = case['n'] ** dim if kind == 'limiting' else math.prod(_cells(case))
        nbytes, flops = _dg_work(dim, order)
        if kind == 'traversal':  # lduh and the face fluxes are results too
            nbytes += 8 * 5 * ((order + 1) ** dim + 2 * dim * (order + 1) ** (dim - 1))
        return dict(bytes=cells * nbytes, flops=cells * flops)
    if kind == 'ensemble':
        w = [(n * n,) + _dg_work(2, o) for o, n in _mix(case)]
        return dict(bytes=case['steps'] * sum(c * b for c, b, _ in w), flops=case['steps'] * sum(c * f for c, _, f in w))
    if kind == 'serving':
        dg, fv = _mix(case)
        w = [(n * n,) + _dg_work(2, o) for o, n in dg]
        cells = 3 * sum(n * n for n in fv)
        return dict(bytes=sum(c * b for c, b, _ in w) + 80 * cells,
                    flops=sum(c * f for c, _, f in w) + _FV_FLOPS[2, 1] * cells)
    if kind == 'fv':
        cells = case['patch'] ** 2
        return dict(bytes=80 * cells, flops=_FV_FLOPS[2, case['scheme']] * cells)
    if kind == 'patches':
        cells = case['count'] * case['patch'] ** case['dim']
        padded = case['count'] * (case['patch'] + 2 * (case['scheme'] + 1)) ** case['dim']
        return dict(bytes=80 * padded, flops=_FV_FLOPS[case['dim'], case['scheme']] * cells)
    dim, b, s = case['dim'], case['order'] + 1, 2 * case['order'] + 1
    sweep = sum(2 * 5 * b * s ** (k + 1) * b ** (dim - 1 - k) for k in range(dim))
    back = sum(2 * 5 * s * b ** (k + 1) * s ** (dim - 1 - k) for k in range(dim))
    lobatto = dim * 2 * 5 * b * b ** dim
    nbytes = 8 * 5 * (2 * b ** dim + 2 * s ** dim) + 16 * 5 * (2 * dim + 2)
    return dict(bytes=case['count'] * nbytes, flops=case['count'] * (sweep + back + sweep + lobatto))


# ------------------------------------------------------------------ 64-bit values
def _lagrange(nodes, x):
    """phi_i(x) and phi_i'(x) of the Lagrange basis on `nodes`: arrays [len(nodes), len(x)]."""
    n, x = len(nodes), np.atleast_1d(np.asarray(x, dtype=np.float64))
    val, der = np.ones((n, len(x))), np.zeros((n, len(x)))
    for i in range(n):
        for j in range(n):
            if j != i:
                val[i] *= (x - nodes[j]) / (nodes[i] - nodes[j])
        for k in range(n):
            if k != i:
                t = np.ones(len(x)) / (nodes[i] - nodes[k])
                for j in range(n):
                    if j not in (i, k):
                        t = t * (x - nodes[j]) / (nodes[i] - nodes[j])
                der[i] += t
    return val, der


class _Basis:
    def __init__(self, order):
        x, w = _nodes(order)
        left, right = _lagrange(x, 0.0)[0][:, 0], _lagrange(x, 1.0)[0][:, 0]
        der = _lagrange(x, x)[1]                      # der[p, l] = phi_p'(x_l)
        kxi = der * w[None, :]                        # kxi[p, l] = int phi_p' phi_l
        ik1 = np.linalg.inv(np.outer(right, right) - kxi)
        t = dict(w=w, der=der.T, time=ik1 * w[None, :], start=ik1 @ left, left=left, right=right, kxi=kxi)
        for k, v in t.items():
            setattr(self, k, torch.as_tensor(np.ascontiguousarray(v), device='cuda'))


def _along(m, f, axis):
    """sum_p m[i, p] f[.., p at axis, ..]"""
    return torch.movedim(torch.tensordot(f, m, dims=([axis], [1])), -1, axis)


def _pressure(q):
    return (GAMMA - 1) * (q[..., 4] - 0.5 * (q[..., 1] ** 2 + q[..., 2] ** 2 + q[..., 3] ** 2) / q[..., 0])


def _flux(q, d):
    p, u = _pressure(q), q[..., d + 1] / q[..., 0]
    f = u[..., None] * q
    f[..., d + 1] += p
    f[..., 4] += u * p
    return f


def _speed(q, d):
    """largest |u - c|, |u|, |u + c|; |u| alone where the pressure is negative (an overshoot at a discontinuity)"""
    u, c = q[..., d + 1] / q[..., 0], torch.sqrt(GAMMA * _pressure(q) / q[..., 0])
    return u.abs() + torch.nan_to_num(c, nan=0.0)


def _cell_dt(u, dim, order, dx):
    """stable dt of each cell: u [cells, nodes, 5], dx [cells or 1, dim]"""
    den = sum(_speed(u, d) / dx[:, d, None] for d in range(dim))
    return _dt_factor(order) / den.max(1).values


def _node_axes(dim, d, lead):
    """axis of direction d in [lead.., (z,) y, x, 5]"""
    return lead + dim - 1 - d


def _predict(u, dim, t, dx, dt):
    """Space-time predictor and volume integral of cells u [c, (z,) y, x, 5] with per-cell dx [c, dim] and dt [c]:
    lduh and the faces' states and fluxes [c, 2 dim, face nodes.., 5]."""
    b = t.w.numel()
    col = [-1] + [1] * (dim + 2)
    q = u[:, None].expand((u.shape[0], b) + u.shape[1:]).contiguous()
    f = None
    open_ = torch.ones(u.shape[0], dtype=torch.bool, device='cuda')
    for _ in range(2 * b):
        idx = open_.nonzero()[:, 0]
        if idx.numel() == 0:
            break
        qi = q[idx]
        fi = [_flux(qi, d) for d in range(dim)]
        g = sum(_along(t.der, fi[d], _node_axes(dim, d, 2)) / dx[idx, d].reshape(col) for d in range(dim))
        new = t.start.reshape([1, b] + [1] * (dim + 1)) * u[idx][:, None] - dt[idx].reshape(col) * _along(t.time, g, 1)
        err = (new - qi).square().flatten(1).sum(1)
        q[idx] = new
        if f is None:
            f = [torch.empty_like(u) for _ in range(dim)]
        for d in range(dim):
            f[d][idx] = torch.tensordot(fi[d], t.w, dims=([1], [0]))
        open_[idx] = err >= 1e-14
        del qi, fi, g, new
    qh = torch.tensordot(q, t.w, dims=([1], [0]))
    wn = [t.w.reshape([1] + [-1 if a == dim - 1 - d else 1 for a in range(dim)] + [1]) for d in range(dim)]
    lduh, qs, fs = 0, [], []
    cell = [-1] + [1] * (dim + 1)
    for d in range(dim):
        other = math.prod(wn[e] for e in range(dim) if e != d)
        ax = _node_axes(dim, d, 1)
        lduh = lduh + _along(t.kxi, f[d], ax) * other / dx[:, d].reshape(cell)
        for side in (t.left, t.right):
            qs.append(torch.tensordot(qh, side, dims=([ax], [0])))
            fs.append(torch.tensordot(f[d], side, dims=([ax], [0])))
    return lduh, torch.stack(qs, 1), torch.stack(fs, 1)


def _dg_step(u, dim, order, dx, dt, nb, bc=None):
    """One ADER-DG step of cells u [c, nodes, 5]; nb [c, 2 dim] neighbours (-1: a wall with rule bc[d]).  Returns the new
    state, the increment lduh and the faces' Rusanov fluxes."""
    t, b, c = _Basis(order), order + 1, u.shape[0]
    shape = (b,) * dim + (5,)
    chunk = max(1, (1 << 25) // (b ** (dim + 1) * 5))
    parts = [_predict(u[i:i + chunk].reshape((-1,) + shape), dim, t, dx[i:i + chunk], dt[i:i + chunk])
             for i in range(0, c, chunk)]
    lduh, qb, fb = (torch.cat([p[k] for p in parts]) for k in range(3))
    del parts
    wn = [t.w.reshape([1] + [-1 if a == dim - 1 - d else 1 for a in range(dim)] + [1]) for d in range(dim)]
    wf = t.w.reshape([1, -1, 1]) if dim == 2 else (t.w[:, None] * t.w[None, :]).reshape(1, b, b, 1)
    flux = torch.empty_like(fb)
    cell = [-1] + [1] * dim
    for f in range(2 * dim):
        d, up = f // 2, f & 1
        k = nb[:, f]
        qn, fn = qb[k, f ^ 1], fb[k, f ^ 1]
        wall = k < 0
        if bool(wall.any()):
            qo = qb[wall, f].clone()
            if bc[d] == REFLECT:
                qo[..., d + 1] *= -1.0
                fn[wall] = _flux(qo, d)
            else:
                fn[wall] = fb[wall, f]
            qn[wall] = qo
        mean = [(x * wf).flatten(1, -2).sum(1) for x in (qb[:, f], qn)]
        s = torch.maximum(_speed(mean[0], d), _speed(mean[1], d)).reshape(cell)
        jump = qn - qb[:, f] if up else qb[:, f] - qn
        flux[:, f] = 0.5 * (fb[:, f] + fn) - 0.5 * s * jump
    for d in range(dim):
        other = math.prod(wn[e] for e in range(dim) if e != d)
        ax = _node_axes(dim, d, 1)
        shape_d = [-1 if a == ax else 1 for a in range(dim + 2)]
        lduh = lduh - (flux[:, 2 * d + 1].unsqueeze(ax) * t.right.reshape(shape_d)
                       - flux[:, 2 * d].unsqueeze(ax) * t.left.reshape(shape_d)) * other / dx[:, d].reshape(cell + [1])
    new = u.reshape((-1,) + shape) + dt.reshape(cell + [1]) * lduh / math.prod(wn)
    return new.reshape(u.shape), lduh, flux


def _grid_neighbours(n, bc):
    dim = len(n)
    idx = torch.arange(math.prod(n), device='cuda').reshape(n[::-1])
    nb = []
    for d in range(dim):
        for up in (0, 1):
            k = torch.roll(idx, -1 if up else 1, dim - 1 - d).clone()
            if bc[d]:
                k.select(dim - 1 - d, n[d] - 1 if up else 0).fill_(-1)
            nb.append(k.reshape(-1))
    return torch.stack(nb, 1)


def _exact_grid(case, seed):
    dim, order, n = case['dim'], case['order'], _cells(case)
    bc = [case['bcx'], case['bcy'], case['bcz']][:dim]
    u = _dg_state(case, seed)
    dx = torch.full((u.shape[0], dim), 1.0 / n[0], device='cuda', dtype=torch.float64)
    dt = _cell_dt(u, dim, order, dx).min().expand(u.shape[0])
    return _dg_step(u, dim, order, dx, dt, _grid_neighbours(n, bc), bc)[0].reshape(-1)


def _exact_traversal(case, seed):
    dim, order, n = case['dim'], case['order'], _cells(case)
    u = _dg_state(case, seed)
    dx = torch.full((u.shape[0], dim), 1.0 / n[0], device='cuda', dtype=torch.float64)
    dt = 0.7 * _cell_dt(u, dim, order, dx).min().expand(u.shape[0])
    new, lduh, flux = _dg_step(u, dim, order, dx, dt, _faces(case)[3])
    return dict(luh=new.reshape(-1), lduh=lduh.reshape(-1), fluxes=flux.reshape(-1), dt=_cell_dt(new, dim, order, dx))


def _solves(mix, amps, steps):
    """States of independent 2D density-wave solves on the unit square after `steps` steps, in the order of `mix`."""
    out = [None] * len(mix)
    for order in sorted({o for o, _ in mix}):
        which = [i for i, (o, _) in enumerate(mix) if o == order]
        u, nb, solve, dx, base = [], [], [], [], 0
        for k, i in enumerate(which):
            n = mix[i][1]
            x, y = _node_coordinates(2, order, [n, n], [1.0, 1.0])
            rho = 1.0 + amps[i] * torch.sin(2 * math.pi * (x + y))
            u.append(_conserved(rho, torch.ones_like(rho), 1.0, 1.0).reshape(n * n, -1, 5))
            nb.append(_grid_neighbours([n, n], [0, 0]) + base)
            solve.append(torch.full((n * n,), k, device='cuda', dtype=torch.int64))
            dx.append(torch.full((n * n, 2), 1.0 / n, device='cuda', dtype=torch.float64))
            base += n * n
        u, nb, solve, dx = (torch.cat(v) for v in (u, nb, solve, dx))
        for _ in range(steps):
            least = torch.full((len(which),), math.inf, device='cuda', dtype=torch.float64)
            least.scatter_reduce_(0, solve, _cell_dt(u, 2, order, dx), 'amin')
            u = _dg_step(u, 2, order, dx, least[solve], nb)[0]
        for k, i in enumerate(which):
            out[i] = u[solve == k].reshape(-1)
    return out


def _exact_ensemble(case, seed):
    mix = _mix(case)
    return torch.cat(_solves(mix, _amplitudes(len(mix), seed), case['steps']))


def _minmod(a, b):
    return torch.where(a * b < 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _fv_update(u, dim, ghost, scheme, h, dt):
    """The update of padded patches u [p, (z,) y, x, 5] (cell size h per direction): the new patches, with the face
    contributions that the scheme also adds to the first ghost layer, and the admissible dt of each patch."""
    side = u.shape[1]
    patch = side - 2 * ghost
    axis = [dim - d for d in range(dim)]  # of direction d

    def cut(v, d, lo, hi):
        """interior in the other directions, cells lo..hi-1 of the padded range along d"""
        for e in range(dim):
            v = v.narrow(axis[e], lo if e == d else ghost, (hi - lo) if e == d else patch)
        return v

    lower, upper = [], []  # states on the lower / upper side of each ring cell, per direction
    for d in range(dim):
        mid = cut(u, d, ghost - 1, ghost + patch + 1)
        if scheme == 0:
            lower.append(mid)
            upper.append(mid)
            continue
        slope = _minmod(cut(u, d, ghost, ghost + patch + 2) - mid, mid - cut(u, d, ghost - 2, ghost + patch))
        lower.append(mid - 0.5 * slope)
        upper.append(mid + 0.5 * slope)
    if scheme == 1:
        inner = [(lo.narrow(axis[d], 1, patch), up.narrow(axis[d], 1, patch))
                 for d, (lo, up) in enumerate(zip(lower, upper))]
        rate = 0.5 * dt * sum((_flux(lo, d) - _flux(up, d)) / h[d] for d, (lo, up) in enumerate(inner))
        for d in range(dim):
            lower[d].narrow(axis[d], 1, patch).add_(rate)
            upper[d].narrow(axis[d], 1, patch).add_(rate)
    new, least = u.clone(), None
    for d in range(dim):
        ql, qr = upper[d].narrow(axis[d], 0, patch + 1), lower[d].narrow(axis[d], 1, patch + 1)
        s = torch.maximum(_speed(ql, d), _speed(qr, d))
        f = 0.5 * (_flux(ql, d) + _flux(qr, d)) - 0.5 * s[..., None] * (qr - ql)
        cut(new, d, ghost - 1, ghost + patch).sub_(dt / h[d] * f)
        cut(new, d, ghost, ghost + patch + 1).add_(dt / h[d] * f)
        c = (CFL if scheme == 0 else 0.99) / dim * h[d] / s.flatten(1).max(1).values
        least = c if least is None else torch.minimum(least, c)
    return new, least


def _fv_step(u, patch, ghost, scheme):
    """One step of a periodic 2D patch u [1, S, S, 5] on the unit square; its ghost cells stay as they are."""
    inner = u[:, ghost:-ghost, ghost:-ghost]
    h = 1.0 / patch
    dt = min(float((CFL / 2 * h / _speed(inner, d)).min()) for d in (0, 1))
    p = inner
    for a in (1, 2):
        p = torch.cat([p.narrow(a, patch - ghost, ghost), p, p.narrow(a, 0, ghost)], a)
    out = u.clone()
    out[:, ghost:-ghost, ghost:-ghost] = _fv_update(p, 2, ghost, scheme, [h, h], dt)[0][:, ghost:-ghost, ghost:-ghost]
    return out


def _exact_fv(case, seed):
    ghost = case['scheme'] + 1
    u = _fv_state(2, case['patch'], ghost, 1, seed, True)
    return _fv_step(u, case['patch'], ghost, case['scheme']).reshape(-1)


def _exact_serving(case, seed):
    dg, fv = _mix(case)
    amps = _amplitudes(len(dg) + len(fv), seed)
    out = _solves(dg, amps, 1)
    for n, a in zip(fv, amps[len(dg):]):
        x = (torch.arange(n + 4, device='cuda', dtype=torch.float64) - 1.5) / n
        rho = 1.0 + a * torch.sin(2 * math.pi * (x[None, None, :] + x[None, :, None]))
        u = _conserved(rho, torch.ones_like(rho), 1.0, 1.0)
        for _ in range(3):
            u = _fv_step(u, n, 2, 1)
        out.append(u.reshape(-1))
    return out


def _exact_patches(case, seed):
    dim, patch, ghost, scheme = case['dim'], case['patch'], case['scheme'] + 1, case['scheme']
    u = _fv_state(dim, patch, ghost, case['count'], seed, False)
    chunk = max(1, (1 << 22) // (patch + 2 * ghost) ** dim)
    parts = [_fv_update(u[i:i + chunk], dim, ghost, scheme, [1.0 / patch] * dim, 0.05 / patch)
             for i in range(0, u.shape[0], chunk)]
    return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])


class _Subcells:
    """1D limiter operators of order N: subcell means, the mean-preserving least-squares inverse, Lobatto values."""

    def __init__(self, order):
        x, w = _nodes(order)
        s = 2 * order + 1
        means = np.zeros((s, order + 1))
        for k in range(s):
            means[k] = (_lagrange(x, (k + x) / s)[0] * w[None, :]).sum(1)
        k = np.zeros((order + 2, order + 2))
        k[:-1, :-1] = 2.0 * means.T @ means
        k[:-1, -1] = k[-1, :-1] = w
        back = np.linalg.solve(k, np.vstack([2.0 * means.T, np.full((1, s), 1.0 / s)]))[:-1]
        p = np.polynomial.legendre.Legendre.basis(order)
        lob = (np.concatenate([[-1.0], np.sort(p.deriv().roots().real), [1.0]]) + 1) / 2
        lobatto = _lagrange(x, lob)[0].T
        self.means, self.back, self.lobatto = (torch.as_tensor(np.ascontiguousarray(v), device='cuda')
                                               for v in (means, back, lobatto))


def _tensor_apply(m, v, dim):
    for a in range(1, dim + 1):
        v = _along(m, v, a)
    return v


def _extrema(u, dim, t):
    """per-cell minima and maxima [c, 5] over nodes, Lobatto points and subcell means of u [c, (z,) y, x, 5]"""
    pts = torch.cat([v.flatten(1, -2) for v in (u, _tensor_apply(t.lobatto, u, dim), _tensor_apply(t.means, u, dim))], 1)
    return pts.min(1).values, pts.max(1).values


def _dmp(lo, hi, mn, mx, relaxation=1e-4, scaling=1e-3):
    """verdict per cell, from bounds [c, faces, 5] and the cell's extrema, and the bounds' own extrema over the faces"""
    blo, bhi = lo.min(1).values, hi.max(1).values
    margin = ((bhi - blo) * scaling).clamp_min(relaxation)
    return ~((mn < blo - margin) | (mx > bhi + margin)).any(1), blo, bhi


def _exact_limiter(case, seed):
    dim, order, count = case['dim'], case['order'], case['count']
    b, s, t = order + 1, 2 * order + 1, _Subcells(order)
    u = _uniform(seed, (count, b ** dim, 5), 0.5, 2.0).reshape((count,) + (b,) * dim + (5,))
    lo = _uniform(seed + 1, (count, 2 * dim, 5), 0.1, 0.5)
    hi = _uniform(seed + 2, (count, 2 * dim, 5), 2.0, 2.4)
    mn, mx = _extrema(u, dim, t)
    _, blo, bhi = _dmp(lo, hi, mn, mx)
    lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1] = mn, mx, blo, bhi
    fine = _tensor_apply(t.means, u, dim)
    lim = torch.nn.functional.pad(fine, (0, 0) + (1, 1) * dim)
    return None, lo, hi, lim.reshape(count, -1), _tensor_apply(t.back, fine, dim).reshape(count, -1, 5)


def _exact_limiting(case, seed):
    dim, order, n = case['dim'], case['order'], case['n']
    b, s, t = order + 1, 2 * order + 1, _Subcells(order)
    u = _explosion(case, seed)
    shape = (-1,) + (b,) * dim + (5,)
    dx = torch.full((u.shape[0], dim), 1.0 / n, device='cuda', dtype=torch.float64)
    dt = _cell_dt(u, dim, order, dx).min()
    nb = _grid_neighbours([n] * dim, [0] * dim)
    mn, mx = _extrema(u.reshape(shape), dim, t)
    lo = torch.minimum(mn[:, None], mn[nb])
    hi = torch.maximum(mx[:, None], mx[nb])
    new = _dg_step(u, dim, order, dx, dt.expand(u.shape[0]), nb)[0]
    ok = _dmp(lo, hi, *_extrema(new.reshape(shape), dim, t))[0]
    ok &= ((new[..., 0] > 0) & (_pressure(new) > 0)).all(1)
    status = torch.where(ok, 0, 5)
    for _ in range(4):
        status = torch.maximum(status, status[nb].max(1).values - 1)
    # finite-volume step on the subcells of the troubled cells and two layers of neighbours
    which = (status >= 3).nonzero()[:, 0]
    own = _tensor_apply(t.means, u[which].reshape(shape), dim)
    pad = torch.nn.functional.pad(own, (0, 0) + (1, 1) * dim)
    for d in range(dim):
        ax = dim - d
        for up in (0, 1):
            other = _tensor_apply(t.means, u[nb[which, 2 * d + up]].reshape(shape), dim)
            ghost = pad.select(ax, s + 1 if up else 0)
            for e in range(dim - 1):
                ghost = ghost.narrow(1 + e, 1, s)
            ghost.copy_(other.select(ax, 0 if up else s - 1))
    stepped = _fv_update(pad, dim, 1, 0, [1.0 / (n * s)] * dim, float(dt))[0]
    for a in range(1, dim + 1):
        stepped = stepped.narrow(a, 1, s)
    new[which] = _tensor_apply(t.back, stepped, dim).reshape(which.numel(), -1, 5)
    return new.reshape(-1)


_EXACT = dict(grid=_exact_grid, traversal=_exact_traversal, ensemble=_exact_ensemble, serving=_exact_serving,
              fv=_exact_fv, patches=_exact_patches, limiting=_exact_limiting, limiter=_exact_limiter)


def exact(case, seed):
    return _EXACT[case['kind']](case, seed)
