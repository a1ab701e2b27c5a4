"""GPU tests of many steps of one universe in one launch (grav_steps, steps.cu): one CTA (up
to 48 bodies, 64 for fewer than eight steps), one cluster (up to 512) and one CTA per SM, at the edges of its row groups,
column blocks and grids.

  - the accelerations of every step against the FP64 oracle on that step's own state,
    per body |a - a_ref| <= 1e-5 sum_j |a_ij| (a pair term carries ~1.5e-6 of FP32 rounding
    and, near-corrected, up to 4.5e-6 from positions beyond the near radius; FP32 partial sums
    of at most 32 terms add less than 1e-6), with pairs 1e-3 apart at |x| ~ 1000 planted;
  - each FP64 update bit for bit from those accelerations (_base_.py:58-62), the stage-1
    positions bit for bit what grav_prepare makes of the final state;
  - K steps in one launch, in several launches, one by one and from a graph: the same bits.
"""

import numpy as np
import pytest
import torch

import oracle
from gravitation_gb300.engine import Engine, STEPS_SINGLE_MAX_N
from gravitation_gb300.scenarios import G_DEFAULT, plummer_pair, uniform_cube

pytestmark = pytest.mark.gpu

TOL = 1e-5
SIZES = [1, 2, 4, 5, 63, 64, 65, 67, 128, 511, 512, 513, 641, 1000, 1217, 2560]
MODES = ['fp32n', 'fp32c']


def planted(n, seed):
    r, v, m = uniform_cube(n, seed=seed)
    rng = np.random.default_rng(seed + 1)
    for i, j in ((3, 9), (17, n - 2), (n // 3, n // 2)):
        if 0 <= i < j < n:
            r[i] = np.sign(r[i]) * 990.0 + rng.uniform(-5, 5, 3)
            r[j] = r[i] + rng.uniform(-1e-3, 1e-3, 3)
    return r, v, m


def magnitudes(r, gm):
    out = np.zeros(len(gm))
    for i in range(0, len(gm), 256):
        d2 = ((r[None, :, :] - r[i:i + 256, None, :]) ** 2).sum(-1)
        with np.errstate(divide='ignore'):
            out[i:i + 256] = np.where(d2 > 0, gm[None, :] / d2, 0.0).sum(1)
    return out


def check_steps(mode, n, steps, T=1.0):
    r, v, m = planted(n, 40 + n)
    gm = G_DEFAULT * m
    eng = Engine([n], T, mode=mode)
    assert eng.chained
    eng.set_state(r, v, gm)
    acc = torch.full((steps, n, 4), 7.0, dtype=torch.float64, device=eng.device)
    eng.steps_to(acc)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    acc = acc.cpu().numpy()
    assert np.all(acc[:, :, 3] == 0.0)
    for k in range(steps):
        a = acc[k, :, :3]
        ref = oracle.accel_fp64(r, gm, 1.0, coincident=True)
        err = np.linalg.norm(a - ref, axis=1)
        scale = magnitudes(r, gm)
        assert np.all(err <= TOL * scale), (mode, n, k, np.max(err / np.maximum(scale, 1e-300)))
        r, v = oracle.stage2_fp64(r, v, a, T)
    assert np.array_equal(eng.r[:n, :3].cpu().numpy(), r)
    assert np.array_equal(eng.v[:n, :3].cpu().numpy(), v)
    assert np.array_equal(eng.r[:n, 3].cpu().numpy(), gm)
    pos = eng.pos.clone()
    eng.prepare()
    torch.cuda.synchronize()
    assert torch.equal(pos, eng.pos)


@pytest.mark.parametrize('mode', MODES)
@pytest.mark.parametrize('n', SIZES)
def test_steps_against_oracle(gpu, mode, n):
    check_steps(mode, n, 3)


@pytest.mark.parametrize('mode,n', [('fp32n', 8200), ('fp32n', 6000), ('fp32n', 7500),
                                    ('fp32n', 12288), ('fp32c', 6144), ('fp32un', 5000),
                                    ('fp32cu', 4999)])
def test_steps_large(gpu, mode, n):
    """Near the largest sizes."""
    check_steps(mode, n, 2)


@pytest.mark.parametrize('mode', MODES)
@pytest.mark.parametrize('n', [1, 64, 100, 512, 515, 2000])
def test_steps_split_and_replayed(gpu, mode, n):
    assert n <= STEPS_SINGLE_MAX_N
    r, v, m = planted(n, 8)
    gm = G_DEFAULT * m
    engines = [Engine([n], 1e3, mode=mode) for _ in range(5)]
    for e in engines:
        e.set_state(r, v, gm)
    engines[0].step(6)
    engines[1].step(2)
    engines[1].step(4)
    for _ in range(6):
        engines[2].step(1)
    g = engines[3].capture_graph(3)
    g.replay()
    g.replay()
    engines[4].step(1)
    engines[4].forces()
    engines[4].step(5, write_a=True)
    torch.cuda.synchronize()
    for e in engines:
        e.raise_on_device_error()
        assert torch.equal(engines[0].r, e.r) and torch.equal(engines[0].v, e.v)
        assert torch.equal(engines[0].pos, e.pos)


@pytest.mark.parametrize('mode', MODES)
@pytest.mark.parametrize('n', [50, 300, 1500])
def test_forces_leave_the_state(gpu, mode, n):
    r, v, m = planted(n, 5)
    eng = Engine([n], 1e3, mode=mode)
    eng.set_state(r, v, G_DEFAULT * m)
    before = [x.clone() for x in (eng.r, eng.v, eng.pos)]
    a = eng.forces().clone()
    two = Engine([n], 1e3, mode=mode, fused=False)
    assert not two.chained
    two.set_state(r, v, G_DEFAULT * m)
    b = two.forces().clone()
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(before, (eng.r, eng.v, eng.pos)))
    scale = torch.tensor(magnitudes(r, G_DEFAULT * m), device=a.device)
    assert float(((a - b).norm(dim=1) / scale).max()) < 2e-5


@pytest.mark.parametrize('mode', MODES)
@pytest.mark.parametrize('n', [48, 49, 57, 64])
def test_steps_one_cta_or_cluster(gpu, mode, n):
    """Eight steps of 49 to 64 bodies run in a cluster, fewer in one CTA: the same bits."""
    check_steps(mode, n, 8)
    r, v, m = planted(n, 9)
    one, two = (Engine([n], 1e3, mode=mode) for _ in range(2))
    for e in (one, two):
        e.set_state(r, v, G_DEFAULT * m)
    one.step(8)
    two.step(7)
    two.step(1)
    torch.cuda.synchronize()
    assert torch.equal(one.r, two.r) and torch.equal(one.v, two.v) and torch.equal(one.pos, two.pos)


@pytest.mark.parametrize('n', [48, 64, 500, 1000])
def test_steps_clump(gpu, n):
    """40 bodies within 1e-3 of one another at |x| ~ 1000: a lane meets several near pairs in
    one block of columns, with both of its rows and both columns of a packed pair."""
    r, v, m = uniform_cube(n, seed=n)
    rng = np.random.default_rng(n)
    r[n // 5:n // 5 + 38] = np.array([990.0, -985.0, 991.0]) + rng.uniform(-1e-3, 1e-3, (38, 3))
    r[[0, n - 1]] = r[n // 5] + np.array([[5e-4, 3e-4, 0.0], [-2e-4, 0.0, 4e-4]])
    gm = G_DEFAULT * m
    eng = Engine([n], 1.0, mode='fp32n')
    eng.set_state(r, v, gm)
    acc = torch.zeros((2, n, 4), dtype=torch.float64, device=eng.device)
    eng.steps_to(acc)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    acc = acc.cpu().numpy()
    for k in range(2):
        ref = oracle.accel_fp64(r, gm, 1.0, coincident=True)
        err = np.linalg.norm(acc[k, :, :3] - ref, axis=1)
        assert np.all(err <= TOL * magnitudes(r, gm)), (n, k)
        r, v = oracle.stage2_fp64(r, v, acc[k, :, :3], 1.0)


def spread_groups(n):
    """A cube whose every few groups of four rows hold three bodies on its faces and a heavy one
    at |x| ~ 100, these in pairs 6 apart: (r, v, m, heavy rows)."""
    r, v, m = uniform_cube(n, seed=n)
    rng = np.random.default_rng(n + 1)
    count = min(64, n // 32 * 2)
    groups = np.arange(1, n // 4)[::max(1, (n // 4 - 1) // count)][:count]
    for k in groups:
        r[4 * k:4 * k + 4] = rng.uniform(-1000.0, 1000.0, (4, 3))
        r[4 * k + np.arange(4), rng.integers(0, 3, 4)] = rng.choice([-1.0, 1.0], 4) * rng.uniform(980.0, 1000.0, 4)
    heavy = 4 * groups + rng.integers(0, 4, len(groups))
    for i, j in zip(heavy[::2], heavy[1::2]):
        d = rng.normal(size=3)
        mid = rng.choice([-1.0, 1.0], 3) * rng.uniform(98.0, 101.0, 3)
        mid[rng.permutation(3)[:2]] *= rng.uniform(-0.3, 0.3, 2)
        r[i], r[j] = mid + 3.0 * d / np.linalg.norm(d), mid - 3.0 * d / np.linalg.norm(d)
    m[heavy] = 1e5 * rng.uniform(1.0, 2.0, len(heavy))
    return r, v, m, heavy


@pytest.mark.parametrize('mode,n', [('fp32un', 300), ('fp32un', 2500), ('fp32un', 6000), ('fp32n', 4100),
                                    ('fp32n', 5003)])
def test_steps_shared_radius(gpu, mode, n):
    """Where the pair kernels' rows share a near radius, a group of four consecutive rows does.
    The heavy pairs stand beyond their own radius of 5, where rounding the positions to FP32 alone
    puts their forces 0.6-1.0e-6 off (rms, from the inputs in FP64), and within their group's 49,
    where the rounding of an FP32 pair term is left: three products and the cube of a reciprocal
    square root good to 1.2e-7, at most 5e-7."""
    r, v, m, heavy = spread_groups(n)
    gm = G_DEFAULT * m
    eng = Engine([n], 1.0, mode=mode)
    assert eng.chained
    eng.set_state(r, v, gm)
    acc = torch.zeros((2, n, 4), dtype=torch.float64, device=eng.device)
    eng.steps_to(acc)
    torch.cuda.synchronize()
    eng.raise_on_device_error()
    acc = acc.cpu().numpy()
    for k in range(2):
        ref = oracle.accel_fp64(r, gm, 1.0, coincident=True)
        err = np.linalg.norm(acc[k, heavy, :3] - ref[heavy], axis=1) / np.linalg.norm(ref[heavy], axis=1)
        assert np.sqrt((err ** 2).mean()) < 5e-7, (mode, n, k)
        r, v = oracle.stage2_fp64(r, v, acc[k, :, :3], 1.0)


@pytest.mark.parametrize('mode,n', [('fp32un', 40), ('fp32un', 500), ('fp32un', 3000), ('fp32un', 6144),
                                    ('fp32n', 5003)])
@pytest.mark.parametrize('shape', ['pair', 'steep'])
def test_steps_dense(gpu, shape, mode, n):
    """Two dense spheres, and bodies spread over four decades of distance: near pairs everywhere
    within the radius that a group shares, so that its rows go on with their own."""
    if shape == 'pair':
        r, v, m = plummer_pair(n, seed=n)
    else:
        rng = np.random.default_rng(n)
        u = rng.normal(size=(n, 3))
        r = 10.0 ** rng.uniform(0.0, 4.0, (n, 1)) * u / np.linalg.norm(u, axis=1, keepdims=True)
        v, m = rng.normal(size=(n, 3)), rng.uniform(1.0, 100.0, n)
    gm = G_DEFAULT * m
    one, two = (Engine([n], 1e-3, mode=mode) for _ in range(2))
    for e in (one, two):
        assert e.chained
        e.set_state(r, v, gm)
    acc = torch.zeros((3, n, 4), dtype=torch.float64, device=one.device)
    one.steps_to(acc)
    for _ in range(3):
        two.step(1)
    torch.cuda.synchronize()
    for e in (one, two):
        e.raise_on_device_error()
    if n <= STEPS_SINGLE_MAX_N:
        assert torch.equal(one.r, two.r) and torch.equal(one.v, two.v)
    acc = acc.cpu().numpy()
    for k in range(3):
        ref = oracle.accel_fp64(r, gm, 1.0, coincident=True)
        err = np.linalg.norm(acc[k, :, :3] - ref, axis=1)
        assert np.all(err <= TOL * magnitudes(r, gm)), (shape, n, k)
        r, v = oracle.stage2_fp64(r, v, acc[k, :, :3], 1e-3)


@pytest.mark.parametrize('mode,n', [('fp32n', 100), ('fp32n', 3000), ('fp32un', 5000)])
def test_stage2_after_forces(gpu, mode, n):
    """forces() and then stage2() is a step over the same partial sums as stage1() and stage2()."""
    r, v, m = planted(n, 12)
    a, b = (Engine([n], 1e3, mode=mode) for _ in range(2))
    for e in (a, b):
        assert e.chained
        e.set_state(r, v, G_DEFAULT * m)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for _ in range(2):
        a.forces(stream=side)
        a.stage2(stream=side)
        b.stage1()
        b.stage2()
    torch.cuda.synchronize()
    for e in (a, b):
        e.raise_on_device_error()
    assert torch.equal(a.r, b.r) and torch.equal(a.v, b.v) and torch.equal(a.pos, b.pos)
    assert not np.array_equal(a.r[:n, :3].cpu().numpy(), r)
