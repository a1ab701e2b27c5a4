"""Failure detection without a GPU fault: a device-side wait that expires is reported to
the host through the device error flag, the host raises, and the context stays usable.
(Argument errors are covered on the CPU in test_abi_cpu.py: they are rejected before any
launch.)"""

import ctypes
import time

import numpy as np
import pytest
import torch

import oracle
from gravitation_gb300 import _lib
from gravitation_gb300.engine import Engine
from gravitation_gb300.scenarios import G_DEFAULT, uniform_cube

pytestmark = pytest.mark.gpu


def test_expired_wait_is_reported_and_context_survives(gpu):
    L = _lib.load()
    r, v, m = uniform_cube(500, seed=4)
    eng = Engine([500], 1e3, mode='fp32u')
    eng.set_state(r, v, G_DEFAULT * m)
    s = torch.cuda.current_stream()
    t0 = time.perf_counter()
    _lib.check(L.grav_wait_check(eng.err.data_ptr(), 50_000_000, ctypes.c_void_p(s.cuda_stream)))
    assert eng.device_error() == _lib.GRAV_DEV_TIMEOUT
    assert time.perf_counter() - t0 < 10.0
    with pytest.raises(_lib.GravError, match='bounded wait'):
        eng.raise_on_device_error()
    assert eng.device_error() == _lib.GRAV_DEV_OK          # cleared by the raise
    # the context is still usable: a normal step gives correct forces
    a = eng.forces().cpu().numpy()
    eng.raise_on_device_error()
    ref = oracle.accel_fp64(r.astype(np.float32).astype(np.float64),
                            (G_DEFAULT * m).astype(np.float32).astype(np.float64), 1.0,
                            coincident=True)
    assert oracle.rel_err_per_body(a, ref).max() < 1e-5


def test_wait_check_rejects_bad_arguments(gpu):
    L = _lib.load()
    assert L.grav_wait_check(None, 1000, None) == _lib.GRAV_E_ARG
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    assert L.grav_wait_check(err.data_ptr(), 0, None) == _lib.GRAV_E_ARG
    assert L.grav_wait_check(err.data_ptr(), 3_000_000_000, None) == _lib.GRAV_E_ARG


@pytest.mark.parametrize('sizes,kw', [((64, 4096), {}), ((300, 2000, 9000), {}),
                                      ((33, 500, 4000), {'fused': (1024, 1024)})])
def test_threads_launch_one_kernel_with_different_sizes(gpu, sizes, kw):
    """A kernel's shared-memory limit is not lowered by one thread under another's launch: threads
    stepping universes of different sizes get the states of the steps taken alone."""
    import threading
    states, engines, failed = [], [], []
    for n in sizes:
        r, v, m = uniform_cube(n, seed=n)
        pair = [Engine([n], 1e3, mode='fp32n', **kw) for _ in range(2)]
        for e in pair:
            e.set_state(r, v, G_DEFAULT * m)
        engines.append(pair)
    for alone, _ in engines:
        for _ in range(200):
            alone.step(2)
    torch.cuda.synchronize()
    start = threading.Barrier(len(sizes))

    def work(eng, stream):
        try:
            start.wait()
            for _ in range(200):
                eng.step(2, stream=stream)
            stream.synchronize()
        except Exception as e:   # noqa: BLE001 -- reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(pair[1], torch.cuda.Stream())) for pair in engines]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not failed and not any(t.is_alive() for t in threads), failed
    for alone, threaded in engines:
        threaded.raise_on_device_error()
        assert torch.equal(alone.r, threaded.r) and torch.equal(alone.v, threaded.v)


def test_expired_word_wait_ends_the_others(gpu):
    """64 words per thread that nothing publishes, after one mbarrier: with a limit of 0.2 s the
    CTA waits 0.4 s in all, not 13."""
    L = _lib.load()
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    s = torch.cuda.current_stream()
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    e0.record(s)
    _lib.check(L.grav_wait_check(err.data_ptr(), 200_000_000, ctypes.c_void_p(s.cuda_stream)))
    e1.record(s)
    e1.synchronize()
    assert int(err.item()) == _lib.GRAV_DEV_TIMEOUT
    assert 390.0 < e0.elapsed_time(e1) < 1000.0
