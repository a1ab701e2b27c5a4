"""CPU tests of the engines' host side: what is handed to the kernels, and which plans are
taken, without a GPU."""

import ctypes
import types

import pytest
import torch

from gravitation_gb300 import _lib
from gravitation_gb300 import build as gbuild
from gravitation_gb300.adjoint import AdjointEngine
from gravitation_gb300.engine import (Engine, fitting_tiles, fp64_pair_tile, pair_plan_fits,
                                      plan_fits, plan_part_bytes, tile_list)


@pytest.fixture(scope='module', autouse=True)
def lib():
    gbuild.build()


@pytest.mark.parametrize('steps', [1, 2, 5])
def test_adjoint_steps_hands_over_the_stored_rows(steps):
    """Without a chained launch every backward step reads the caller's own accelerations, the
    last first, on the stream given."""
    eng = AdjointEngine.__new__(AdjointEngine)
    eng.chained, eng.sizes = False, [3]
    eng.device = torch.device('cpu')
    seen = []
    eng.step = lambda stream=None, a_in=None: seen.append((stream, a_in.data_ptr()))
    a = torch.arange(steps * 12, dtype=torch.float64).reshape(steps, 3, 4)
    eng.steps(a, stream='s')
    assert seen == [('s', a[k].data_ptr()) for k in reversed(range(steps))]


GB300_BUDGET = 284208 * 2 ** 20 // 8


@pytest.mark.parametrize('sizes', [[1 << 21], [1 << 22], [3000000], [2000000] * 3, [1 << 24]])
def test_workloads_too_large_for_unique_pairs(sizes):
    """More slots than a plan can number: the FP64 engine takes ordered pairs, and no unique-pair
    plan fits."""
    assert fp64_pair_tile(sizes, 152, GB300_BUDGET) is None
    if sizes[0] == 1 << 24:
        assert pair_plan_fits(sizes, GB300_BUDGET, mode='fp32un') is False


@pytest.mark.parametrize('mode', ['fp32un', _lib.GRAV_MODE_FP64U])
@pytest.mark.parametrize('sizes', [[0], [1], [31], [32, 33, 0, 900], [5000], [70001]])
def test_plan_fits_agrees_with_the_plan(mode, sizes):
    for t in tile_list(mode):
        t.grid = 608
        need = plan_part_bytes(sizes, t, mode)
        assert plan_fits(sizes, t, mode, need) and plan_fits(sizes, t, mode, None)
        assert not need or not plan_fits(sizes, t, mode, need - 1)
    assert len(fitting_tiles(sizes, 'fp32un', 1 << 40)) == len(tile_list('fp32un'))


def test_row_arguments_are_checked():
    """Accelerations whose address goes to a kernel: shape, type, device, and for results the
    layout, before anything is launched."""
    good = torch.zeros((3, 5, 4), dtype=torch.float64)
    bad = [good.to(torch.float32), good[:, :4], good[:, :, :3], good[0], good.tolist(),
           torch.zeros((3, 5, 5), dtype=torch.float64), good.to('meta')]
    adj = AdjointEngine.__new__(AdjointEngine)
    adj.chained, adj.sizes, adj.device = False, [2, 3], torch.device('cpu')
    eng = Engine.__new__(Engine)
    eng.info, eng.device, eng.chained = types.SimpleNamespace(n_bodies=5), torch.device('cpu'), True
    eng._steps = adj.step = None   # a launch would raise TypeError
    for a in bad:
        for call in (adj.steps, eng.steps_to):
            with pytest.raises(ValueError):
                call(a)
    for a in (good.transpose(0, 1).contiguous().transpose(0, 1), good[:1].expand(3, 5, 4),
              torch.zeros((3, 4, 5), dtype=torch.float64).transpose(1, 2)):
        with pytest.raises(ValueError):
            eng.steps_to(a)
    eng.steps_to(good[:0])
    adj.steps(good[:0])


def test_adjoint_steps_of_strided_rows():
    """Rows of a step that are not contiguous are copied; steps that are not are not."""
    eng = AdjointEngine.__new__(AdjointEngine)
    eng.chained, eng.sizes, eng.device = False, [3], torch.device('cpu')
    seen = []
    eng.step = lambda stream=None, a_in=None: seen.append(a_in.clone())
    base = torch.arange(48, dtype=torch.float64)
    for a in (base.reshape(4, 4, 3).transpose(1, 2), base.reshape(4, 3, 4)[::2],
              base[:12].reshape(1, 3, 4).expand(4, 3, 4)):
        del seen[:]
        eng.steps(a)
        assert all(x.is_contiguous() for x in seen)
        assert torch.equal(torch.stack(seen), a.flip(0))


@pytest.mark.parametrize('n', [100, 5000])
def test_no_steps_launch_nothing(n):
    """step(0), and a count below zero as range() takes it."""
    eng = Engine.__new__(Engine)
    eng.chained, eng.fused, eng.sizes = True, None, [n]
    eng._h = lambda stream: None
    eng._steps = None   # a launch would raise TypeError
    for k in (0, -1):
        eng.step(k)


def test_scratch_of_the_many_step_launches_is_aligned():
    """Their exchange uses 128-bit accesses: scratch off a 16-byte boundary is refused."""
    L = _lib.load()
    b = _lib.Batch()
    b.mode = _lib.GRAV_MODE_FP32N
    b.tile = _lib.Tile(1, 128, 128, 1)
    b.n_seg, b.n_pad_total, b.n_bodies, b.n_univ = 1, 128, 100, 1
    b.univ = b.seg = b.pos = b.r = b.v = b.err = 16
    b.eps2 = 1e-25
    a = _lib.Adjoint()
    flat = _lib.Batch.from_buffer_copy(b)
    flat.mode = _lib.GRAV_MODE_FP32
    a.b = ctypes.pointer(flat)
    a.gr = a.gv = a.ggm = a.upos = a.part7 = a.a_in = 16
    for off in (8, 24, 4):
        scratch = ctypes.c_void_p(off)   # never dereferenced: validation fails first
        assert L.grav_steps(ctypes.byref(b), 1, 0, 0, scratch, None) == _lib.GRAV_E_ARG
        assert L.grav_adjoint_steps(ctypes.byref(a), 0, 0, scratch, None) == _lib.GRAV_E_ARG
    scratch = ctypes.c_void_p(32)
    assert L.grav_steps(ctypes.byref(b), 1, 0, 0, scratch, None) == _lib.GRAV_OK           # no steps
    assert L.grav_adjoint_steps(ctypes.byref(a), 0, 0, scratch, None) == _lib.GRAV_OK
