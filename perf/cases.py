"""The measured cases: the steps, forces and gradients that a user of the framework runs.

Sizes and distributions are the repository's own workloads: one universe of 2^4 .. 2^17
bodies in a uniform cube (the sweep of bench.py), the precision stress of two Plummer
spheres, batches of universes of log-uniform size, the differentiable rollout, and the
kernel package's step as a front end drives it.  The precision mode is the one the package
picks for float32 or float64 at that size unless a case names another.

Kinds of case
  step      Engine, `steps` full steps (stage 1 + stage 2) on the device state, either
            replayed from a CUDA graph of that many steps or launched; returns r and v
  batch     the same for many universes in one Engine
  forces    accelerations alone, on the engine or through the allocation-free entry point;
            kept in float32, the precision the FP32 modes compute them in
  rollout   gradients of a fit to observed final positions with respect to r0, v0 and
            float32 masses, by autograd through the differentiable rollout
  frontend  gb1.universe.step(): one synchronous step with the state in host memory
"""

import ctypes
import math

import numpy as np
import torch

from gravitation_gb300 import _lib
from gravitation_gb300.adjoint import Rollout, rollout
from gravitation_gb300.engine import Engine
from gravitation_gb300.kernel.gb1 import universe
from gravitation_gb300.plugin import default_mode

G = 6.6740831e-11   # the reference's constant
T = 1.0e3           # and time step


def listed():
    return [
        # what a front end does with a small float32 universe: step() and read the bodies
        {'name': 'frontend_1024', 'kind': 'frontend', 'n': 1024},
        # the smallest simulations: a graph of many steps, latency is all of it
        {'name': 'step_64', 'kind': 'step', 'n': 64, 'steps': 20, 'graph': True},
        # a small ragged universe, its steps launched one after another
        {'name': 'step_1000', 'kind': 'step', 'n': 1000, 'steps': 20, 'graph': False},
        # mid sizes of the sweep
        {'name': 'step_4096', 'kind': 'step', 'n': 4096, 'steps': 20, 'graph': True},
        {'name': 'step_16384', 'kind': 'step', 'n': 16384, 'steps': 1, 'graph': True},
        # the headline single universe, and the largest of the sweep
        {'name': 'step_65536', 'kind': 'step', 'n': 65536, 'steps': 1, 'graph': False},
        {'name': 'step_131072', 'kind': 'step', 'n': 131072, 'steps': 1, 'graph': False},
        # dense clusters: double-single separations for every pair
        {'name': 'plummer_16384', 'kind': 'step', 'n': 16384, 'steps': 1, 'graph': True,
         'shape': 'plummer'},
        # dtype='float64', odd size
        {'name': 'float64_8191', 'kind': 'step', 'n': 8191, 'steps': 1, 'graph': False,
         'dtype': 'float64'},
        # forces for a caller with an integrator of its own
        {'name': 'forces_6000', 'kind': 'forces', 'n': 6000, 'noalloc': False},
        # 256 universes of 64 .. 16384 bodies
        {'name': 'batch_256', 'kind': 'batch', 'n_univ': 256, 'n_min': 64, 'n_max': 16384,
         'sizes_seed': 1, 'steps': 1, 'graph': True},
        # forward and backward of the differentiable rollout
        {'name': 'rollout_4096', 'kind': 'rollout', 'n': 4096, 'steps': 64, 'every': 32},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['step', 'step', 'step', 'batch', 'forces', 'rollout', 'frontend'])
    if kind == 'step':
        option = rng.choice(['float32', 'float32', 'float32', 'plummer', 'float64', 'mode'])
        hi = {'float64': 12000, 'plummer': 32768}.get(option, 120000)
        n = _log_uniform(rng, 16, hi)
        case = {'kind': 'step', 'n': n, 'steps': 20 if n < 4608 else 1,
                'graph': rng.random() < 0.5}
        if option == 'plummer':
            case['shape'] = 'plummer'
        elif option == 'float64':
            case.update(dtype='float64', steps=1)
        elif option == 'mode':
            case['mode'] = rng.choice(['fp32', 'fp32u', 'fp32c', 'fp32cu', 'fp32n', 'fp32un'])
            if case['mode'] not in ('fp32u', 'fp32un'):
                case['n'] = n = min(n, 70000)
        return case
    if kind == 'batch':
        n_min = _log_uniform(rng, 16, 512)
        return {'kind': 'batch', 'n_univ': _log_uniform(rng, 2, 200), 'n_min': n_min,
                'n_max': _log_uniform(rng, 2 * n_min, 16384),
                'sizes_seed': rng.randrange(1 << 20), 'steps': 1, 'graph': rng.random() < 0.5}
    if kind == 'forces':
        noalloc = rng.random() < 0.5
        return {'kind': 'forces', 'n': _log_uniform(rng, 64, 16384 if noalloc else 65536),
                'noalloc': noalloc}
    if kind == 'rollout':
        n = _log_uniform(rng, 128, 12288)
        return {'kind': 'rollout', 'n': n, 'every': rng.choice([5, 8, 32]),
                'steps': max(8, min(96, int(1.2e9 / (n * n))))}
    return {'kind': 'frontend', 'n': _log_uniform(rng, 16, 16384)}


# ---- inputs ---------------------------------------------------------------------------
def _cube(n, rng):
    """Positions U[-1000, 1000]^3, velocities N(0, 1), masses U[1, 100]."""
    return rng.uniform(-1e3, 1e3, (n, 3)), rng.normal(0.0, 1.0, (n, 3)), rng.uniform(1.0, 100.0, n)


def _plummer(n, rng, a=50.0, sep=1000.0, vrel=5.0):
    """Two Plummer spheres approaching along x, masses log-uniform in [0.1, 1000]."""
    m = np.exp(rng.uniform(math.log(0.1), math.log(1000.0), n))
    rad = a / np.sqrt(rng.uniform(1e-6, 0.999, n) ** (-2.0 / 3.0) - 1.0)
    u = rng.normal(0.0, 1.0, (n, 3))
    r = rad[:, None] * u / np.linalg.norm(u, axis=1, keepdims=True)
    vesc = np.sqrt(2.0 * G * 0.5 * m.sum() / a) * (1.0 + (rad / a) ** 2) ** -0.25
    v = rng.normal(0.0, 0.3, (n, 3)) * vesc[:, None]
    side = np.where(np.arange(n) < n - n // 2, -1.0, 1.0)
    r[:, 0] += 0.5 * sep * side
    v[:, 0] -= 0.5 * vrel * side
    return r, v, m


def _sizes(case):
    if case['kind'] != 'batch':
        return [case['n']]
    rng = np.random.default_rng(case['sizes_seed'])
    s = np.exp(rng.uniform(math.log(case['n_min']), math.log(case['n_max']), case['n_univ']))
    return [int(x) for x in np.clip(np.rint(s), case['n_min'], case['n_max'])]


def _inputs(case, seed):
    """(r, v, m) of all bodies, universe after universe."""
    rng = np.random.default_rng(seed)
    make = _plummer if case.get('shape') == 'plummer' else _cube
    parts = [make(n, rng) for n in _sizes(case)]
    return tuple(np.concatenate(x) for x in zip(*parts))


def _mode(case, sizes, r):
    if case.get('mode'):
        return case['mode']
    if case['kind'] == 'batch':
        return 'fp32un' if max(sizes) >= 4608 else 'fp32n'
    return default_mode(case.get('dtype', 'float32'), sizes[0], r=r)


def _observed(r, v, steps, seed):
    """Final positions as observed: the bodies' free paths with an error of 10 units."""
    rng = np.random.default_rng([seed, 1])
    return r + steps * T * v + rng.normal(0.0, 10.0, r.shape)


# ---- a pass ---------------------------------------------------------------------------
def prepare(case, seed):
    sizes = _sizes(case)
    r, v, m = _inputs(case, seed)
    kind = case['kind']
    state = {'kind': kind, 'n': len(m)}
    if kind == 'frontend':
        u = universe(T=T, G=G, dtype='float32', autotune=False)
        for i in range(len(m)):
            u.add_object(name='', r=list(r[i]), v=list(v[i]), m=float(m[i]))
        u.start()
        first = next(iter(u))
        # the rows of all bodies' positions and velocities, as pm._r and pm._v view them
        state.update(u=u, r=first._r.base, v=first._v.base)
        return state
    if kind == 'rollout':
        dev = torch.device('cuda', torch.cuda.current_device())
        state.update(
            r0=torch.tensor(r, device=dev, requires_grad=True),
            v0=torch.tensor(v, device=dev, requires_grad=True),
            m=torch.tensor(m, dtype=torch.float32, device=dev, requires_grad=True),
            seen=torch.tensor(_observed(r, v, case['steps'], seed), device=dev),
            steps=case['steps'], every=case['every'],
            ro=Rollout(sizes, T, case['steps'], case['every']))
        return state
    if kind == 'forces' and case['noalloc']:
        rows = torch.tensor(np.concatenate([r, (G * m)[:, None]], axis=1), device='cuda')
        state.update(lib=_lib.load(), rows=rows, out=torch.empty_like(rows),
                     err=torch.zeros(1, dtype=torch.int32, device='cuda'),
                     max_gm=float((G * m).max()))
        return state
    eng = Engine(sizes, T, mode=_mode(case, sizes, r))
    eng.set_state(r, v, G * m)
    state['eng'] = eng
    if kind != 'forces':
        state['steps'] = case['steps']
        state['graph'] = eng.capture_graph(case['steps']) if case['graph'] else None
    return state


def run(state):
    kind = state['kind']
    if kind == 'frontend':
        state['u'].step()
        return {'r': state['r'], 'v': state['v']}
    if kind == 'rollout':
        rK, vK = rollout(state['r0'], state['v0'], state['m'], G, T, state['steps'],
                         state['every'], ro=state['ro'])
        loss = ((rK - state['seen']) ** 2).sum(1).mean()
        g = torch.autograd.grad(loss, (state['r0'], state['v0'], state['m']))
        return {'r': rK.detach(), 'v': vK.detach(), 'g_r': g[0], 'g_v': g[1], 'g_m': g[2]}
    if kind == 'forces':
        if 'lib' in state:
            stream = torch.cuda.current_stream().cuda_stream
            _lib.check(state['lib'].grav_forces_noalloc(
                ctypes.c_void_p(state['rows'].data_ptr()),
                ctypes.c_void_p(state['out'].data_ptr()), state['n'], state['max_gm'],
                ctypes.c_void_p(state['err'].data_ptr()), ctypes.c_void_p(stream)))
            return state['out'][:, :3].to(torch.float32)
        return state['eng'].forces().to(torch.float32)
    if state['graph'] is not None:
        state['graph'].replay()
    else:
        state['eng'].step(state['steps'])
    n = state['n']
    return {'r': state['eng'].r[:n], 'v': state['eng'].v[:n]}


def work(case):
    """Each unordered pair once: 3 subtractions, 3 multiply-adds, a reciprocal square root,
    4 products and 6 multiply-adds (26 operations); its transpose in the backward sweep: 13
    multiply-adds, 14 other operations and the same 14 up to r^-3 again (54)."""
    sizes = _sizes(case)
    pairs = sum(n * (n - 1) // 2 for n in sizes)
    bodies = sum(sizes)
    if case['kind'] == 'forces':
        return {'bytes': bodies * (32 + 12), 'flops': 26 * pairs}
    if case['kind'] == 'rollout':
        return {'bytes': bodies * 8 * 26, 'flops': (26 + 54) * pairs * case['steps']}
    return {'bytes': bodies * 128, 'flops': 26 * pairs * case.get('steps', 1)}


# ---- the same in 64 bits -----------------------------------------------------------------
def _pair_blocks(r):
    """Row blocks (rows, d = r_j - r_i, 1/|d|^3 with 0 at zero separation)."""
    n = r.shape[0]
    rows = max(1, min(n, (1 << 26) // n))
    for i in range(0, n, rows):
        d = r[None, :, :] - r[i:i + rows, None, :]
        r2 = (d * d).sum(-1)
        inv = torch.where(r2 > 0, torch.rsqrt(r2), torch.zeros_like(r2))
        yield slice(i, min(n, i + rows)), d, inv


def _accel(r, gm):
    a = torch.empty_like(r)
    for s, d, inv in _pair_blocks(r):
        a[s] = torch.einsum('ij,ijc->ic', inv ** 3 * gm[None, :], d)
    return a


def _transposed(r, gm, u):
    """h = J_A(r)^T u and g_i = sum_j u_j . d / |d|^3 for d = r_j - r_i."""
    h, g = torch.empty_like(r), torch.empty_like(gm)
    for s, d, inv in _pair_blocks(r):
        inv3 = inv ** 3
        duj, dui = torch.einsum('ijc,jc->ij', d, u), torch.einsum('ijc,ic->ij', d, u[s])
        q = 3.0 * (gm[s, None] * duj - gm[None, :] * dui) * inv3 * inv * inv
        h[s] = (gm[s, None] * (inv3 @ u) - u[s] * (inv3 @ gm)[:, None]
                - torch.einsum('ij,ijc->ic', q, d))
        g[s] = (duj * inv3).sum(1)
    return h, g


def exact(case, seed):
    sizes = _sizes(case)
    r, v, m = _inputs(case, seed)
    dev = torch.device('cuda', torch.cuda.current_device())
    r, v, gm = (torch.tensor(x, device=dev) for x in (r, v, G * m))
    if case['kind'] == 'forces':
        return _accel(r, gm)
    steps = case.get('steps', 1)
    if case['kind'] == 'rollout':
        seen = torch.tensor(_observed(r.cpu().numpy(), v.cpu().numpy(), steps, seed), device=dev)
        gm = (G * torch.tensor(m, dtype=torch.float32, device=dev)).to(torch.float64)
        path = []
        for _ in range(steps):
            path.append(r)
            v = v + T * _accel(r, gm)
            r = r + T * v
        g_r = (2.0 / len(m)) * (r - seen)
        g_v, g_gm = torch.zeros_like(g_r), torch.zeros_like(gm)
        for rk in reversed(path):
            u = g_v + T * g_r
            h, g = _transposed(rk, gm, u)
            g_r, g_v, g_gm = g_r + T * h, u, g_gm - T * g
        return {'r': r, 'v': v, 'g_r': g_r, 'g_v': g_v, 'g_m': G * g_gm}
    at = np.concatenate([[0], np.cumsum(sizes)])
    for _ in range(steps):
        a = torch.cat([_accel(r[i:j], gm[i:j]) for i, j in zip(at[:-1], at[1:])])
        v = v + T * a
        r = r + T * v
    zero = torch.zeros_like(gm)
    return {'r': torch.cat([r, gm[:, None]], 1), 'v': torch.cat([v, zero[:, None]], 1)}
