"""GPU tests of many backward steps of one universe in one launch (grav_adjoint_steps,
adjoint_steps.cu) at the edges of its row groups, column blocks and grids.

  - gradients against FP64 sums over all ordered pairs, step by step, on positions that FP32
    holds exactly: a pair's terms carry at most ~3e-6 of FP32 rounding (inv^5 of an
    approximate reciprocal square root, three products of three terms), FP32 partial sums of at
    most 32 terms less than 2e-6, both of the sum of the terms' magnitudes, so TOL = 1e-5;
  - the reversed state bit for bit from the separately rounded FP64 products and sums, the
    prepared FP32 positions and u bit for bit from the final state;
  - K steps in one launch, in several and from a graph: the same bits;
  - against the same steps of two launches each.
"""

import numpy as np
import pytest
import torch

from gravitation_gb300.adjoint import AdjointEngine
from gravitation_gb300.scenarios import G_DEFAULT

pytestmark = pytest.mark.gpu

TOL = 1e-5


def pair_sums(r, gm, u):
    """(h, g, magnitudes of their terms) in FP64; coincident bodies do not act on each other."""
    n = len(gm)
    h, g = np.zeros((n, 3)), np.zeros(n)
    mh, mg = np.zeros(n), np.zeros(n)
    un = np.linalg.norm(u, axis=1)
    for a in range(0, n, 128):
        s = slice(a, min(a + 128, n))
        d = r[None, :, :] - r[s, None, :]
        d2 = (d * d).sum(-1)
        inv = np.where(d2 > 0, 1.0 / np.sqrt(np.where(d2 > 0, d2, 1.0)), 0.0)
        inv3 = inv ** 3
        duj = (d * u[None, :, :]).sum(-1)
        dui = (d * u[s, None, :]).sum(-1)
        t = gm[s, None] * duj - gm[None, :] * dui
        h[s] = (inv3[:, :, None] * (gm[s, None, None] * u[None, :, :] - gm[None, :, None] * u[s, None, :])
                - 3.0 * (t * inv3 * inv * inv)[:, :, None] * d).sum(1)
        g[s] = (duj * inv3).sum(1)
        mh[s] = 4.0 * (inv3 * (gm[s, None] * un[None, :] + gm[None, :] * un[s, None])).sum(1)
        mg[s] = (inv * inv * un[None, :]).sum(1)
    return h, g, mh, mg


def state(n, seed):
    """Positions on a lattice of 2^-6 in [-100, 100]^3 (two coincident), masses, gradients."""
    rng = np.random.default_rng(seed)
    r = rng.integers(-6400, 6401, (n, 3)) / 64.0
    if n > 4:
        r[1] = r[3]
    return r, G_DEFAULT * rng.uniform(1.0, 100.0, n), rng.normal(size=(n, 3)), rng.normal(size=(n, 3))


def load(eng, r, v, gm, gr, gv):
    n = len(gm)
    dev = eng.device
    eng.set_state(torch.tensor(np.column_stack([r, gm]), device=dev),
                  torch.tensor(np.column_stack([v, np.zeros(n)]), device=dev))
    eng.gr[:n, :3] = torch.tensor(gr, device=dev)
    eng.gv[:n, :3] = torch.tensor(gv, device=dev)
    eng.ggm.zero_()
    eng.prepare()


@pytest.mark.parametrize('n,steps', [(n, 3) for n in (1, 2, 4, 5, 63, 64, 65, 130, 511, 512, 513,
                                                      700, 1217, 2560)] + [(4099, 2), (6900, 2)])
def test_adjoint_steps_gradients(gpu, n, steps):
    """At rest and without accelerations the positions stay: every step's sums are exact."""
    r, gm, gr, gv = state(n, n)
    eng = AdjointEngine([n], 1.0)
    assert eng.chained
    load(eng, r, np.zeros((n, 3)), gm, gr, gv)
    eng.steps(torch.zeros((steps, n, 4), dtype=torch.float64, device=eng.device))
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    bound_h, bound_g, ggm = np.zeros(n), np.zeros(n), np.zeros(n)
    for _ in range(steps):
        u = gv + gr
        h, g, mh, mg = pair_sums(r, gm, u)
        gr, gv, ggm = gr + h, u, ggm - g
        bound_h += TOL * mh
        bound_g += TOL * mg
    assert np.all(np.abs(eng.gr[:n, :3].cpu().numpy() - gr).max(1) <= bound_h + 1e-15 * np.abs(gr).max())
    assert np.all(np.abs(eng.ggm[:n].cpu().numpy() - ggm) <= bound_g)
    assert np.allclose(eng.gv[:n, :3].cpu().numpy(), gv, rtol=1e-12, atol=steps * bound_h.max())
    assert np.array_equal(eng.r[:n, :3].cpu().numpy(), r)


@pytest.mark.parametrize('n', [3, 64, 100, 515, 3001])
def test_adjoint_steps_reversal_and_splits(gpu, n):
    r, gm, gr, gv = state(n, 7 + n)
    rng = np.random.default_rng(n)
    v, T = rng.normal(size=(n, 3)), 1.0 / 3.0
    acc = np.zeros((6, n, 4))
    acc[:, :, :3] = rng.normal(size=(6, n, 3))
    engines = [AdjointEngine([n], T) for _ in range(4)]
    a = torch.tensor(acc, device=engines[0].device)
    for e in engines:
        load(e, r, v, gm, gr, gv)
    engines[0].steps(a)
    engines[1].steps(a[2:])
    engines[1].steps(a[:2])
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        engines[2].steps(a)
    graph.replay()
    for k in reversed(range(6)):
        engines[3].step(a_in=a[k])
    torch.cuda.synchronize()
    for e in engines:
        e.raise_on_device_error()
    for k in reversed(range(6)):
        r = r - T * v
        v = v - T * acc[k, :, :3]
    one = engines[0]
    assert np.array_equal(one.r[:n, :3].cpu().numpy(), r)
    assert np.array_equal(one.v[:n, :3].cpu().numpy(), v)
    for e in engines[1:3]:
        for x in ('r', 'v', 'gr', 'gv', 'ggm'):
            assert torch.equal(getattr(e, x), getattr(one, x)), x
        assert torch.equal(e.pos[:4 * n], one.pos[:4 * n])
        assert torch.equal(e.upos[:4 * n], one.upos[:4 * n])
    two = engines[3]
    assert torch.equal(two.r, one.r) and torch.equal(two.v, one.v)
    assert torch.equal(two.pos[:4 * n], one.pos[:4 * n])
    for x, tol in (('gr', 1e-9), ('gv', 1e-9), ('ggm', 1e-4)):
        p, q = getattr(one, x)[:n], getattr(two, x)[:n]
        assert float((p - q).norm()) <= tol * float(q.norm()), x


def test_adjoint_steps_choice(gpu):
    """A given tile or kernel, a batch and sizes that do not fit keep two launches per step."""
    assert not AdjointEngine([700], 1.0, pairs=True).chained
    assert not AdjointEngine([700], 1.0, tile=(1, 128, 128)).chained
    assert not AdjointEngine([300, 400], 1.0).chained
    assert not AdjointEngine([9000], 1.0).chained


@pytest.mark.parametrize('sizes,pairs', [([700], True), ([700], False), ([300, 450], None),
                                         ([7300], None)])
def test_adjoint_steps_unchained_on_another_stream(gpu, sizes, pairs):
    """Two launches per step on a stream that is not the current one: the bits of the steps one
    by one, and no memory taken."""
    n = sum(sizes)
    r, gm, gr, gv = state(n, 3)
    v = np.random.default_rng(4).normal(size=(n, 3))
    engines = [AdjointEngine(sizes, 0.5, pairs=pairs) for _ in range(2)]
    a = torch.randn((4, n, 4), dtype=torch.float64, device=engines[0].device)
    a[:, :, 3] = 0.0
    for e in engines:
        assert not e.chained
        load(e, r, v, gm, gr, gv)
    for k in reversed(range(4)):
        engines[0].step(a_in=a[k])
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    engines[1].steps(a, stream=side)
    assert torch.cuda.max_memory_allocated() == before
    torch.cuda.synchronize()
    engines[1].raise_on_device_error()
    for x in ('r', 'v', 'gr', 'gv', 'ggm', 'pos', 'upos'):
        assert torch.equal(getattr(engines[0], x), getattr(engines[1], x)), x


@pytest.mark.parametrize('sizes', [[70], [600], [300, 200]])
def test_adjoint_steps_layouts(gpu, sizes):
    """Steps apart by more than their rows, one step's rows repeated and strided rows: the bits of
    the same accelerations packed."""
    n = sum(sizes)
    r, gm, gr, gv = state(n, 5)
    a = torch.randn((8, n, 4), dtype=torch.float64, device='cuda')
    for strided in (a[::2], a[:1].expand(3, n, 4), a.transpose(1, 2).contiguous().transpose(1, 2)):
        engines = [AdjointEngine(sizes, 0.5) for _ in range(2)]
        for e, x in zip(engines, (strided, strided.clone(memory_format=torch.contiguous_format))):
            load(e, r, np.ones((n, 3)), gm, gr, gv)
            e.steps(x)
            e.raise_on_device_error()
        for x in ('r', 'v', 'gr', 'gv', 'ggm'):
            assert torch.equal(getattr(engines[0], x), getattr(engines[1], x)), x


def test_adjoint_steps_mass_gradient_as_exact_as_two_launches(gpu):
    """The mass gradients' partial sums end every 16 blocks of columns like the others': at the
    largest size the error of the middle body is no higher than the two-launch steps', whose
    partial sums run over one j-tile (10 % for the spread of the median over 6900 bodies)."""
    n = 6900
    rng = np.random.default_rng(0)
    r = rng.integers(-64000, 64001, (n, 3)) / 64.0
    gm = (G_DEFAULT * rng.uniform(1.0, 100.0, n)).astype(np.float32).astype(np.float64)
    u = rng.normal(size=(n, 3)).astype(np.float32).astype(np.float64)
    zero = np.zeros((n, 3))
    h, g, _, _ = pair_sums(r, gm, u)
    _, g2, _, _ = pair_sums(r, gm, u + h)
    ref = -(g + g2)
    engines = [AdjointEngine([n], 1.0) for _ in range(2)]
    a = torch.zeros((2, n, 4), dtype=torch.float64, device='cuda')
    for e in engines:
        load(e, r, zero, gm, zero, u)
    engines[0].steps(a)
    for k in (1, 0):
        engines[1].step(a_in=a[k])
    one, two = (np.median(np.abs(e.ggm.cpu().numpy() - ref) / np.abs(ref)) for e in engines)
    assert one <= 1.1 * two, (one, two)
