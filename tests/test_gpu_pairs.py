"""GPU tests of the packed unique-pair kernels (stage1_sym.cu) at the edges of their tiles:
every compiled shape of every unique-pair mode with one body below, at and above one row
block, with several blocks and a ragged end, and with pairs of bodies 1e-3 apart at
|x| ~ 1000 planted inside a block and across blocks (the near correction's row and column
terms).

Tolerance, per body: |a - a_ref| <= 1e-5 sum_j |a_ij|, a_ij the pair terms in FP64.  A pair
term carries the rounding of the FP32 operations that form it (about ten, each 2^-24, and
the reciprocal square root's 2^-22 three times: below 1.5e-6) and, in fp32un, up to 4.5e-6
from the rounding of positions beyond the near radius; the FP32 partial sums of at most 256
terms add less than 2e-6 (random rounding signs).
"""

import numpy as np
import pytest

import oracle
from gravitation_gb300 import _lib
from gravitation_gb300.engine import Engine, tile_list
from gravitation_gb300.scenarios import G_DEFAULT, plummer_pair, uniform_cube

pytestmark = pytest.mark.gpu

TOL = 1e-5


def planted_cube(n, rows, seed):
    """A uniform cube with close pairs: within the first block and from the first to the
    last body's block."""
    r, v, m = uniform_cube(n, seed=seed)
    rng = np.random.default_rng(seed + 1)
    for k in range(6):
        for i, j in ((7 + 40 * k, 23 + 40 * k), (11 + 40 * k, n - 3 - 5 * k)):
            if max(i, j) < n and i < min(rows, n) and j > i:
                r[i] = np.sign(r[i]) * 990.0 + rng.uniform(-5, 5, 3)
                r[j] = r[i] + rng.uniform(-1e-3, 1e-3, 3)
    if n > 6:
        r[5] = [0.02, -0.01, 0.03]     # where padding rows must not be met as near
    return r, v, m


def magnitudes(r, gm):
    """sum_j Gm_j / |r_j - r_i|^2 per body."""
    out = np.zeros(len(gm))
    for i in range(0, len(gm), 256):
        d2 = ((r[None, :, :] - r[i:i + 256, None, :]) ** 2).sum(-1)
        with np.errstate(divide='ignore'):
            out[i:i + 256] = np.where(d2 > 0, gm[None, :] / d2, 0.0).sum(1)
    return out


@pytest.mark.parametrize('mode', ['fp32u', 'fp32cu', 'fp32un'])
@pytest.mark.parametrize('case', ['below', 'block', 'above', 'ragged'])
def test_pair_tiles_at_block_edges(gpu, mode, case):
    done = {}
    for t in tile_list(mode):
        rows = t.bpt * t.threads
        n = {'below': rows - 1, 'block': rows, 'above': rows + 1,
             'ragged': 2 * rows + t.jtile + 33}[case]
        if n not in done:
            r, v, m = planted_cube(n, rows, seed=900 + n)
            gm = G_DEFAULT * m
            rr, gg = r, gm
            if mode == 'fp32u':   # plain FP32 separations: on the positions it reads
                rr = r.astype(np.float32).astype(np.float64)
                gg = gm.astype(np.float32).astype(np.float64)
            done[n] = (r, v, gm, oracle.accel_fp64(rr, gg, 1.0, coincident=True),
                       magnitudes(rr, gg))
        r, v, gm, ref, scale = done[n]
        for grid in (0, 5):
            eng = Engine([n], 1e3, mode=mode, tile=_lib.Tile(t.bpt, t.threads, t.jtile, grid))
            eng.set_state(r, v, gm)
            a = eng.forces().cpu().numpy()
            eng.raise_on_device_error()
            err = np.linalg.norm(a - ref, axis=1) / scale
            assert err.max() < TOL, (mode, t, grid, n, err.max())


@pytest.mark.parametrize('rows', [32, 64, 128])
def test_fp64_pair_blocks(gpu, rows):
    """The FP64 unique-pair kernel at the edges of its row blocks, close and coincident pairs
    in one block and across blocks: 1e-14 of the pair terms' magnitudes (a term carries about
    ten roundings of 2^-53, a sum of up to 450 terms the root of their number)."""
    for n in (1, 31, rows - 1, rows, rows + 1, 3 * rows + 33):
        r, v, m = planted_cube(n, rows, seed=700 + n)
        if n > rows + 20:
            r[rows + 17] = r[5]
        gm = G_DEFAULT * m
        ref, scale = oracle.accel_fp64(r, gm, 1.0, coincident=True), magnitudes(r, gm)
        for grid in (0, 5):
            eng = Engine([n], 1e3, mode=_lib.GRAV_MODE_FP64U, tile=_lib.Tile(1, rows, 32, grid))
            assert eng.mode_name == 'fp64'
            eng.set_state(r, v, gm)
            a = eng.forces().cpu().numpy()
            eng.raise_on_device_error()
            err = np.linalg.norm(a - ref, axis=1)
            assert np.all(err <= 1e-14 * scale), (rows, n, grid, np.max(err / np.maximum(scale, 1e-300)))


def test_fp64_scratch_limits(gpu):
    """Separations outside the fast reciprocal's range (and huge ones) follow the law: two
    bodies 1e-120, 1e-60, 1e60 and 1e150 apart, and the default engine takes unique pairs."""
    for d in (1e-120, 1e-60, 1.0, 1e60, 1e150):
        r = np.array([[0.0, 0, 0], [d, 0, 0]])
        gm = np.array([2.0, 3.0]) * d * d      # accelerations 3 and -2
        eng = Engine([2], 1.0, mode='fp64')
        assert eng.mode == _lib.GRAV_MODE_FP64U
        eng.set_state(r, np.zeros((2, 3)), gm)
        a = eng.forces().cpu().numpy()
        ordered = Engine([2], 1.0, mode='fp64', tile=_lib.Tile(1, 128, 128, 0))
        ordered.set_state(r, np.zeros((2, 3)), gm)
        b = ordered.forces().cpu().numpy()
        assert np.array_equal(np.isfinite(a), np.isfinite(b)), d
        if 1e-100 < d < 1e100:
            assert np.allclose(a, [[3.0, 0, 0], [-2.0, 0, 0]], rtol=1e-15), (d, a)


@pytest.mark.parametrize('mode', ['fp32n', 'fp32un'])
def test_near_modes_with_escaped_bodies(gpu, mode):
    """Rows far out test apart from the others of their thread, each against its own near
    radius: one escaped body, two that are near each other, and a thread whose rows are mostly
    such."""
    n = 2100
    rng = np.random.default_rng(3)
    r = rng.uniform(-1e3, 1e3, (n, 3))
    m = rng.uniform(1.0, 100.0, n)
    r[5] = [2e6, -1e6, 5e5]
    r[700], r[1500] = [-3e5, 2e5, 1e5], [-3e5 + 0.5, 2e5, 1e5 + 0.25]
    r[64:64 + 256] *= 40.0
    r[900], r[901] = 0.0, [0.0, 1e-3, -2e-3]     # at the origin and next to it
    gm = G_DEFAULT * m
    ref = oracle.accel_fp64(r, gm, 1.0, coincident=True)
    scale = magnitudes(r, gm)
    for t in tile_list(mode):
        eng = Engine([n], 1.0, mode=mode, tile=t, fused=False)
        eng.set_state(r, np.zeros((n, 3)), gm)
        a = eng.forces().cpu().numpy()
        eng.raise_on_device_error()
        err = np.linalg.norm(a - ref, axis=1) / scale
        assert err.max() < TOL, (t.key(), int(err.argmax()), err.max())


def test_near_mode_in_dense_clusters(gpu):
    """Two Plummer spheres away from the origin: most j-tiles meet so many near pairs that they
    run on double-single separations, in diagonal blocks too.  Two bodies closer than the FP32
    resolution of their coordinates contribute nothing to each other there either."""
    n = 3000
    r, _, m = plummer_pair(n, seed=4)
    r[40] = np.float32(r[40]).astype(np.float64)
    same = r.copy()
    r[41], same[41] = r[40] + 1e-9, r[40]
    gm = G_DEFAULT * m
    ref = oracle.accel_fp64(same, gm, 1.0, coincident=True)
    scale = magnitudes(same, gm)
    for t in tile_list('fp32un'):
        eng = Engine([n], 1.0, mode='fp32un', tile=t, fused=False)
        eng.set_state(r, np.zeros((n, 3)), gm)
        a = eng.forces().cpu().numpy()
        eng.raise_on_device_error()
        assert np.array_equal(a, eng.forces().cpu().numpy())
        err = np.linalg.norm(a - ref, axis=1) / scale
        assert err.max() < TOL, (t.key(), int(err.argmax()), err.max())


@pytest.mark.parametrize('n,one_wave', [(6145, True), (7168, True), (7297, True), (7700, False)])
def test_default_tile_of_one_wave(gpu, n, one_wave):
    """fp32un from 6145 bodies to where a CTA would get a second unit: rows of 4 in blocks of 512;
    its forces like those of any shape."""
    r, v, m = planted_cube(n, 512, n)
    eng = Engine([n], 1.0, mode='fp32un')
    assert (eng.tile.key() == (4, 128, 128)) == one_wave
    assert not one_wave or eng.info.n_units <= eng.info.grid
    eng.set_state(r, v, G_DEFAULT * m)
    a = eng.forces().cpu().numpy()
    eng.raise_on_device_error()
    ref = oracle.accel_fp64(r, G_DEFAULT * m, 1.0, coincident=True)
    assert np.all(np.linalg.norm(a - ref, axis=1) <= TOL * magnitudes(r, G_DEFAULT * m))
