"""GPU tests of the adjoint (csrc/adjoint.cu, gravitation_gb300/adjoint.py).

Gradients of L = mean_i |r_K,i - t_i|^2 with respect to r0, v0 and m, checked against
  - the FP64 oracle's vector-Jacobian product for a single step,
  - autograd through a plain PyTorch FP64 integrator (same law, same update),
  - FP64 central finite differences (eps 1e-6) on 16 seeded coordinates.
The systems used here are compact and slow (velocities ~ the virial speed), so that
gravity, not free streaming, shapes the final state and finite differences in FP64
resolve the mass gradients.
"""

import numpy as np
import pytest
import torch

import oracle
from gravitation_gb300.adjoint import Rollout, rollout, torch_reference_rollout
from gravitation_gb300.scenarios import G_DEFAULT, mass_perturbation, uniform_cube

pytestmark = pytest.mark.gpu

T = 1.0e3


def compact(n, seed):
    # half-width 100: over tens of steps gravity moves bodies by ~0.1, so a 1e-6 change
    # of a mass moves final positions by ~1e-9, far above their FP64 resolution (~1e-14)
    r, v, m = uniform_cube(n, seed=seed, half=100.0, v_sigma=1e-4)
    return r, v, m


def relerr(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize('pairs', [False, True])
@pytest.mark.parametrize('store_a', [False, True])
def test_single_step_against_oracle_vjp(gpu, pairs, store_a):
    """Both backward pair kernels: every ordered pair, and each unordered pair once
    (700 bodies = 3 row blocks of the unique-pair plan, so column slots are used), each
    recomputing the accelerations or taking the forward's (store_a)."""
    n = 700
    r, v, m = compact(n, 3)
    rng = np.random.default_rng(1)
    c = rng.normal(size=(n, 3))
    # the forward in the plain FP32 arithmetic the backward pair kernels recompute with,
    # so that the reversed state can be checked exactly
    ro = Rollout([n], T, 1, every=1, adj_pairs=pairs, store_a=store_a, mode='fp32')
    assert ro.adj.pairs == pairs and ro.store_a == store_a
    dev = torch.device('cuda')
    rK, vK = ro.forward(torch.tensor(r, device=dev), torch.tensor(v, device=dev),
                        torch.tensor(G_DEFAULT * m, device=dev))
    # L = sum c . r_1  ->  gr_1 = c, gv_1 = 0, u = T c
    gr, gv, ggm = ro.backward(torch.tensor(c, device=dev), torch.zeros((n, 3), device=dev,
                                                                        dtype=torch.float64))
    u = T * c
    h, g = oracle.vjp_fp64(r, m, G_DEFAULT, u)
    assert relerr(gr.cpu().numpy(), c + T * h) < 1e-6
    assert relerr(gv.cpu().numpy(), u) < 1e-15
    # dL/dGm = -T g  (g_k = sum_j u_j . (r_j - r_k)/|r_j - r_k|^3)
    assert relerr(ggm.cpu().numpy(), -T * g) < 1e-5
    # the reversed state is the initial state
    r_rev, v_rev = ro.reversed_state
    assert np.max(np.abs(r_rev.cpu().numpy() - r)) <= 1e-12 * np.max(np.abs(r))
    assert np.max(np.abs(v_rev.cpu().numpy() - v)) <= 1e-15 + 1e-9 * np.max(np.abs(v))


@pytest.mark.parametrize('tile', [(2, 256, 64), (2, 128, 64), (4, 128, 128)])
@pytest.mark.parametrize('store_a', [False, True])
def test_single_step_every_unique_pair_tile(gpu, tile, store_a):
    """Every compiled shape of the unique-pair backward kernel (2 rows per thread with the
    compensated sums in registers, 4 with them in shared memory), with and without the
    forward's accelerations, against the oracle's VJP: 1500 bodies, 3 row blocks of 512
    rows at 4 rows per thread, so that column slots are used."""
    from gravitation_gb300.adjoint import AdjointEngine
    n = 1500
    r, v, m = compact(n, 5)
    c = np.random.default_rng(6).normal(size=(n, 3))
    ro = Rollout([n], T, 1, every=1, store_a=store_a, mode='fp32')
    ro.adj = AdjointEngine([n], T, tile=tile, pairs=True)
    dev = torch.device('cuda')
    ro.forward(torch.tensor(r, device=dev), torch.tensor(v, device=dev),
               torch.tensor(G_DEFAULT * m, device=dev))
    gr, gv, ggm = ro.backward(torch.tensor(c, device=dev),
                              torch.zeros((n, 3), device=dev, dtype=torch.float64))
    ro.adj.raise_on_device_error()
    h, g = oracle.vjp_fp64(r, m, G_DEFAULT, T * c)
    assert relerr(gr.cpu().numpy(), c + T * h) < 1e-6
    assert relerr(ggm.cpu().numpy(), -T * g) < 1e-5
    r_rev, _ = ro.reversed_state
    assert np.max(np.abs(r_rev.cpu().numpy() - r)) <= 1e-12 * np.max(np.abs(r))


@pytest.mark.parametrize('store_a', [False, True])
def test_single_step_batch_one_lane_per_row(gpu, store_a):
    """A batch of two universes with more than 16384 padded rows, where the adjoint stage
    2 gives each row one lane instead of splitting it: both universes against the
    oracle's VJP, and the reversed state."""
    sizes = [9000, 8500]
    parts = [compact(n, 20 + i) for i, n in enumerate(sizes)]
    r = np.concatenate([p[0] for p in parts])
    v = np.concatenate([p[1] for p in parts])
    m = np.concatenate([p[2] for p in parts])
    c = np.random.default_rng(4).normal(size=r.shape)
    ro = Rollout(sizes, T, 1, every=1, store_a=store_a, mode='fp32u')
    assert ro.adj.info.n_pad_total > 16384
    dev = torch.device('cuda')
    ro.forward(torch.tensor(r, device=dev), torch.tensor(v, device=dev),
               torch.tensor(G_DEFAULT * m, device=dev))
    gr, gv, ggm = ro.backward(torch.tensor(c, device=dev),
                              torch.zeros(r.shape, device=dev, dtype=torch.float64))
    gr, ggm = gr.cpu().numpy(), ggm.cpu().numpy()
    o = 0
    for (ru, _, mu), n in zip(parts, sizes):
        h, g = oracle.vjp_fp64(ru, mu, G_DEFAULT, T * c[o:o + n])
        assert relerr(gr[o:o + n], c[o:o + n] + T * h) < 1e-6
        # g_k sums ~9000 terms u_j.d/|d|^3 of random sign: FP32 pair terms leave ~1e-5
        # relative error after the cancellation (an indexing fault would be O(1))
        assert relerr(ggm[o:o + n], -T * g) < 3e-5
        o += n
    r_rev, v_rev = ro.reversed_state
    assert np.max(np.abs(r_rev.cpu().numpy() - r)) <= 1e-12 * np.max(np.abs(r))


@pytest.mark.parametrize('every,n,pairs,store_a', [(1, 192, None, None), (8, 192, None, None),
                                                   (40, 192, None, True), (8, 600, True, False),
                                                   (8, 600, True, 'auto'), (13, 600, True, True)])
def test_rollout_against_torch_autograd(gpu, every, n, pairs, store_a):
    steps = 40
    r, v, m = compact(n, 5)
    tgt = r + np.random.default_rng(2).normal(scale=1.0, size=r.shape)
    dev = torch.device('cuda')
    G = G_DEFAULT

    def grads(fn):
        r0 = torch.tensor(r, device=dev, requires_grad=True)
        v0 = torch.tensor(v, device=dev, requires_grad=True)
        mm = torch.tensor(m, device=dev, requires_grad=True)
        rK, vK = fn(r0, v0, mm)
        loss = ((rK - torch.tensor(tgt, device=dev)) ** 2).sum(1).mean()
        loss.backward()
        return [x.grad.cpu().numpy() for x in (r0, v0, mm)], float(loss)

    ro = (Rollout([n], T, steps, every, adj_pairs=pairs, store_a=store_a)
          if pairs is not None or store_a is not None else None)
    ours, l1 = grads(lambda a, b, c: rollout(a, b, c, G, T, steps, every=every, ro=ro))
    ref, l2 = grads(lambda a, b, c: torch_reference_rollout(a, b, c, G, T, steps))
    assert abs(l1 - l2) <= 1e-6 * abs(l2)
    for name, x, y in zip(('r0', 'v0', 'm'), ours, ref):
        assert relerr(x, y) < 1e-5, (name, relerr(x, y))


def test_rollout_against_finite_differences(gpu):
    n, steps = 128, 30
    r, v, m = compact(n, 7)
    f = mass_perturbation(n, 7)
    rt, _ = oracle.rollout_fp64(r, v, m * f, G_DEFAULT, T, steps)   # target run
    dev = torch.device('cuda')
    r0 = torch.tensor(r, device=dev, requires_grad=True)
    v0 = torch.tensor(v, device=dev, requires_grad=True)
    mm = torch.tensor(m, device=dev, requires_grad=True)
    rK, _ = rollout(r0, v0, mm, G_DEFAULT, T, steps, every=8)
    loss = ((rK - torch.tensor(rt, device=dev)) ** 2).sum(1).mean()
    loss.backward()

    def L(rr, vv, mv):
        rk, _ = oracle.rollout_fp64(rr, vv, mv, G_DEFAULT, T, steps)
        return float(((rk - rt) ** 2).sum(1).mean())

    rng = np.random.default_rng(16)
    # central differences with eps = 1e-6 in units of each variable's scale: positions
    # (~100) and masses (~50) take eps = 1e-6 directly; the velocities here are ~1e-4,
    # where 1e-6 would be a 1 % change, so their step is 1e-6 * 1e-3
    eps_of = {0: 1e-6, 1: 1e-9, 2: 1e-6}
    checks = []
    for _ in range(16):
        which = int(rng.integers(3))
        i = int(rng.integers(n))
        c = int(rng.integers(3))
        eps = eps_of[which]
        rp, rm_, vp, vm, mp, mmn = r.copy(), r.copy(), v.copy(), v.copy(), m.copy(), m.copy()
        if which == 0:
            rp[i, c] += eps
            rm_[i, c] -= eps
            g = r0.grad[i, c].item()
        elif which == 1:
            vp[i, c] += eps
            vm[i, c] -= eps
            g = v0.grad[i, c].item()
        else:
            mp[i] += eps
            mmn[i] -= eps
            g = mm.grad[i].item()
        fd = (L(rp, vp, mp) - L(rm_, vm, mmn)) / (2 * eps)
        checks.append((which, g, fd))
    for which, g, fd in checks:
        assert abs(g - fd) <= 1e-4 * abs(fd) + 1e-12, (which, g, fd)


def test_fp64_reference_gradients_match_oracle_adjoint(gpu):
    """The checkpointed PyTorch FP64 autograd reference (used by the adjoint check at
    the full configuration) against the oracle's FP64 discrete adjoint."""
    from gravitation_gb300.adjoint import reference_gradients_fp64
    n, steps = 256, 20
    r, v, m = compact(n, 5)
    t = r + 1.0
    rk, _ = oracle.rollout_fp64(r, v, m, G_DEFAULT, T, steps)
    g = (2.0 / n) * (rk - t)
    want = oracle.adjoint_rollout_fp64(r, v, m, G_DEFAULT, T, steps, g, np.zeros_like(g),
                                       every=6)
    dev = torch.device('cuda')
    tt = lambda x: torch.tensor(x, device=dev)  # noqa: E731
    got = reference_gradients_fp64(tt(r), tt(v), tt(m), G_DEFAULT, T, steps, tt(g),
                                   tt(np.zeros_like(g)), every=6)
    for a, b in zip(got, want):
        assert relerr(a.cpu().numpy(), b) < 1e-12


# the differentiable-rollout configuration (uniform cube N = 4096, seed 3, checkpoint
# every 32), shortened to 64 steps so that the CPU oracle's FP64 adjoint stays within
# seconds; gradients of the mean squared distance to the target made by the same FP64
# run with masses scaled by the seeded factor in [0.99, 1.01].  Errors are
# ||g - g64|| / ||g64|| over every body.  Two tolerances:
#   ADJ_TOL   the adjoint sweep itself, seeded with the exact FP64 dL/dr_K (its pair terms
#             are FP32 on the FP64 state: measured 5e-9, 1e-10, 7e-6 on GB300);
#   E2E_TOL   forward + adjoint, seeded from the rollout's own r_K: the loss is
#             ill-conditioned (r_K - t is ~1e-9 of r_K), so the forward's force error
#             dominates (near-corrected forward: measured 7e-5, 7e-5, 3e-5; plain FP32
#             separations: 1e-3).
ADJ_TOL = {'r0': 1e-7, 'v0': 1e-8, 'm': 5e-5}
E2E_TOL = {'r0': 2e-4, 'v0': 2e-4, 'm': 1e-4}


@pytest.mark.parametrize('store_a', [False, True])
def test_config4_shortened_against_fp64_adjoint(gpu, store_a):
    n, steps, every, seed = 4096, 64, 32, 3
    r, v, m = uniform_cube(n, seed=seed)
    f = mass_perturbation(n, seed)
    t, _ = oracle.rollout_fp64(r, v, m * f, G_DEFAULT, T, steps)
    rk64, _ = oracle.rollout_fp64(r, v, m, G_DEFAULT, T, steps)
    g64 = (2.0 / n) * (rk64 - t)
    want = oracle.adjoint_rollout_fp64(r, v, m, G_DEFAULT, T, steps, g64, np.zeros_like(g64),
                                       every=every)
    dev = torch.device('cuda')
    ro = Rollout([n], T, steps, every, store_a=store_a)
    assert ro.fwd.mode_name == 'fp32n'
    rK, _ = ro.forward(torch.tensor(r, device=dev), torch.tensor(v, device=dev),
                       torch.tensor(G_DEFAULT * m, device=dev))
    seeds = {'exact': g64, 'own': (2.0 / n) * (rK.cpu().numpy() - t)}
    for name, tol in (('exact', ADJ_TOL), ('own', E2E_TOL)):
        g = torch.tensor(seeds[name], device=dev)
        gr, gv, ggm = ro.backward(g, torch.zeros_like(g))
        got = (gr.cpu().numpy(), gv.cpu().numpy(), G_DEFAULT * ggm.cpu().numpy())
        errs = {k: relerr(a, b) for k, a, b in zip(('r0', 'v0', 'm'), got, want)}
        for k, e in errs.items():
            assert e < tol[k], (name, errs)


@pytest.mark.parametrize('graphs', [False, True])
@pytest.mark.parametrize('sizes,adj_pairs', [([500], None), ([300, 200], None), ([500], True)])
def test_rollout_on_another_stream(gpu, graphs, sizes, adj_pairs):
    """forward and backward on a stream that lags behind the current one: the bits of the
    current stream's run, read on the current stream, on first use and on a new state."""
    n, steps = sum(sizes), 7
    dev = torch.device('cuda')
    ros = [Rollout(sizes, T, steps, 3, adj_pairs=adj_pairs, graphs=graphs) for _ in range(2)]
    side = torch.cuda.Stream()
    for seed in (1, 2):
        r, v, m = compact(n, seed)
        r, v, gm = (torch.tensor(x, device=dev) for x in (r, v, G_DEFAULT * m))
        c = torch.tensor(np.random.default_rng(seed).normal(size=(n, 3)), device=dev)
        torch.cuda.synchronize()
        out = []
        for ro, stream in zip(ros, (None, side)):
            if stream is not None:
                with torch.cuda.stream(stream):
                    torch.cuda._sleep(20_000_000)   # ~10 ms
            rK, vK = (x.clone() for x in ro.forward(r, v, gm, stream=stream))
            out.append((rK, vK) + ro.backward(c, torch.zeros_like(c), stream=stream) + ro.reversed_state)
        for x, y in zip(*out):
            assert torch.equal(x, y)
    for ro in ros:
        ro.fwd.raise_on_device_error()
        ro.adj.raise_on_device_error()


@pytest.mark.parametrize('n', [200, 7300])
def test_rollout_reused_with_other_masses(gpu, n):
    """G m of 1e-1, 1e3, 1e-1 in turn: the smallest separation that the kernels resolve (eps2)
    follows the masses of the pass, as in a Rollout made for it, captured or not."""
    steps, dev = 6, torch.device('cuda')
    r, v, m = compact(n, 4)
    r[1] = r[0]             # coincident bodies meet at r2 = eps2
    r[2] = 0.0              # and these between the two passes' eps2
    r[3] = [1e-11, 0.0, 0.0]
    r, v = (torch.tensor(x, device=dev) for x in (r, v))
    ro = Rollout([n], 1e-9, steps, 3)
    eps = []
    for gm in (0.1, 1e3, 1e3, 0.1, 0.1):
        g = torch.tensor(gm * m, device=dev)
        got = [x.clone() for x in ro.forward(r, v, g)]
        eps.append(ro.fwd.batch.eps2)
        want = Rollout([n], 1e-9, steps, 3, graphs=False).forward(r, v, g)
        assert all(torch.isfinite(x).all() for x in got)
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert eps[1] > 10 * eps[0]


def test_rollout_reports_a_forward_timeout(gpu):
    """A device error of the forward, set here from the host, is raised by the backward."""
    from gravitation_gb300 import _lib
    r, v, m = compact(100, 3)
    r0, v0, mm = (torch.tensor(x, device='cuda', requires_grad=True) for x in (r, v, m))
    ro = Rollout([100], T, 4, 2)
    rK, _ = rollout(r0, v0, mm, G_DEFAULT, T, 4, ro=ro)
    ro.fwd.err.fill_(_lib.GRAV_DEV_TIMEOUT)
    with pytest.raises(_lib.GravError, match='bounded wait'):
        rK.sum().backward()
    assert ro.fwd.device_error() == _lib.GRAV_DEV_OK
