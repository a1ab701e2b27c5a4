"""Device engine: FP64 state, work-list plan and stage launches for one or more universes.

PyTorch owns every device buffer; the C ABI (libgravgb300.so) borrows raw pointers.
One ``Engine`` holds a packed batch of universes (a single universe is a batch of
one) and drives the persistent stage-1 kernel and the FP64 stage-2 kernel on a CUDA
stream.  There is no CPU path: without the library or a GB300 every call raises.

Layout in HBM (all packed universe after universe):
  r, v     float64 [n_bodies, 4]   (x, y, z, G*m) and (vx, vy, vz, 0); or, after
           bind_host_state, the caller's pinned host tensors of that layout
  pos      padded stage-1 positions: float4 hi (+ float4 lo in fp32c/fp32cu/fp32n/fp32un)
           or double4
  part     8-byte entries [n_slots, 3, itile]  partial sums written by stage 1: FP32
           (hi, lo) pairs in the row slots (FP64 values in fp64 mode); the unique-pair
           column slots hold FP32 sums in their first half
  univ/seg plan tables (grav_univ_desc / grav_seg_desc)
"""

import ctypes

import numpy as np
import torch

from . import _lib
from ._lib import check

_DEVICE_CACHE = {}


class DeviceInfo:
    def __init__(self, index, sm_count, cc):
        self.index = index
        self.sm_count = sm_count
        self.cc = cc
        self.name = torch.cuda.get_device_name(index)

    def __repr__(self):
        return 'DeviceInfo(%d, %s, sms=%d, cc=%d.%d)' % (
            self.index, self.name, self.sm_count, self.cc[0], self.cc[1])


def device_info(device=None):
    """SM count and compute capability; raises unless the GPU is sm_103 (GB300)."""
    if not torch.cuda.is_available():
        raise RuntimeError('gravitation_gb300 needs a CUDA GPU (GB300); none is visible')
    index = torch.device('cuda', torch.cuda.current_device()).index if device is None else \
        torch.device(device).index
    if index is None:
        index = torch.cuda.current_device()
    if index not in _DEVICE_CACHE:
        L = _lib.load()
        sms, ma, mi = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
        with torch.cuda.device(index):
            check(L.grav_device_query(index, ctypes.byref(sms), ctypes.byref(ma), ctypes.byref(mi)))
        _DEVICE_CACHE[index] = DeviceInfo(index, sms.value, (ma.value, mi.value))
    return _DEVICE_CACHE[index]


def tile_list(mode):
    L = _lib.load()
    m = _lib.MODES[mode] if isinstance(mode, str) else mode
    n = L.grav_tile_list(m, None, 0)
    if n < 0:
        check(n)
    arr = (_lib.Tile * n)()
    L.grav_tile_list(m, arr, n)
    return [_lib.Tile(t.bpt, t.threads, t.jtile, 0) for t in arr]


def occupancy(mode, tile, device=None):
    L = _lib.load()
    m = _lib.MODES[mode] if isinstance(mode, str) else mode
    out = ctypes.c_int32()
    info = device_info(device)
    with torch.cuda.device(info.index):
        check(L.grav_occupancy(m, ctypes.byref(tile), ctypes.byref(out)))
    return out.value


def make_plan(sizes, T, tile, mode='fp32'):
    """Host-side plan (no GPU needed): (PlanInfo, univ ctypes array, seg ctypes array).
    The unique-pair modes (fp32u, fp32cu, fp32un, GRAV_MODE_FP64U) use grav_plan_pairs, the
    others grav_plan."""
    L = _lib.load()
    fn = L.grav_plan_pairs if mode in _lib.PAIR_MODES else L.grav_plan
    sizes = [int(x) for x in sizes]
    nu = len(sizes)
    n_arr = (ctypes.c_int32 * max(nu, 1))(*sizes)
    T_list = list(T) if np.ndim(T) else [float(T)] * nu
    T_arr = (ctypes.c_double * max(nu, 1))(*[float(x) for x in T_list])
    info = _lib.PlanInfo()
    check(fn(nu, n_arr, T_arr, ctypes.byref(tile), ctypes.byref(info), None, None))
    univ = (_lib.UnivDesc * max(info.n_univ, 1))()
    seg = (_lib.SegDesc * max(info.n_seg, 1))()
    check(fn(nu, n_arr, T_arr, ctypes.byref(tile), ctypes.byref(info), univ, seg))
    return info, univ, seg


def plan_part_bytes(sizes, tile, mode, comps=3):
    """Bytes of partial-sum slots the plan of `mode` (all pairs or unique pairs) needs for
    `sizes` with `tile`: grav_part_bytes, scaled to `comps` components per slot entry (3
    for stage 1; the backward pair kernel keeps 7).  Host-side, no GPU needed.

    The unique-pair plan keeps one column slot per pair of row blocks, so its slots grow
    as N^2 / (rows per block): 12.9 GB at N = 2^20 with 1024-row blocks, 206 GB at 2^22.
    The all-pairs plan keeps one slot per CTA piece of a row block: 36 MB at 2^20."""
    L = _lib.load()
    fn = L.grav_plan_pairs if mode in _lib.PAIR_MODES else L.grav_plan
    sizes = [int(x) for x in sizes]
    nu = len(sizes)
    n_arr = (ctypes.c_int32 * max(nu, 1))(*sizes)
    T_arr = (ctypes.c_double * max(nu, 1))(*([1.0] * max(nu, 1)))
    t = _lib.Tile(tile.bpt, tile.threads, tile.jtile, max(int(tile.grid), 1))
    info = _lib.PlanInfo()
    check(fn(nu, n_arr, T_arr, ctypes.byref(t), ctypes.byref(info), None, None))
    return int(L.grav_part_bytes(ctypes.byref(info))) * comps // 3


def plan_fits(sizes, tile, mode, budget, comps=3):
    """True when the unique-pair plan of `mode` with `tile` keeps its partial-sum slots within
    `budget` bytes (None: no limit).  Its column slots, one per pair of row blocks, are
    counted before it is planned: a plan with more slots than its tables can number does not
    fit either."""
    rows = tile.bpt * tile.threads
    blocks = [-(-int(n) // rows) for n in sizes]
    slots = sum(nb * (nb - 1) // 2 + nb for nb in blocks)   # at least; at most a grid's more
    if slots + max(int(tile.grid), 1) > 2 ** 31 - 1:
        return False
    if budget is None:
        return True
    return slots * rows * 8 * comps <= budget and plan_part_bytes(sizes, tile, mode, comps) <= budget


SLOT_BUDGET_FRACTION = 0.125
SLOT_BUDGET_NO_GPU = 32 << 30


def slot_budget_bytes(device=None):
    """Device memory that a unique-pair plan chosen by default may spend on partial-sum
    slots: an eighth of the GPU's memory (about 35 GB on a GB300); 32 GiB when no GPU is
    visible (host-side planning)."""
    if not torch.cuda.is_available():
        return SLOT_BUDGET_NO_GPU
    idx = torch.cuda.current_device() if device is None else torch.device(device).index
    if idx is None:
        idx = torch.cuda.current_device()
    return int(torch.cuda.get_device_properties(idx).total_memory * SLOT_BUDGET_FRACTION)


def fitting_tiles(sizes, mode, budget=None, comps=3, tiles=None):
    """The shapes in `tiles` (default: every compiled shape of `mode`) whose plan keeps
    its partial-sum slots within `budget` bytes (default slot_budget_bytes()); every shape
    in the all-pairs modes, whose slots do not grow with N^2.  The autotuner and the
    default shape choose among these."""
    tiles = list(tile_list(mode) if tiles is None else tiles)
    if mode not in _lib.PAIR_MODES:
        return tiles
    if budget is None:
        budget = slot_budget_bytes()
    return [t for t in tiles if plan_fits(sizes, t, mode, budget, comps)]


def pair_plan_fits(sizes, budget=None, mode='fp32u', comps=3, tiles=None):
    """True when some shape in `tiles` (default: every compiled shape of `mode`) keeps the
    unique-pair plan's slots within `budget` bytes (default slot_budget_bytes()); the
    autotuner and the default shape then pick only such shapes (fitting_tiles)."""
    return len(fitting_tiles(sizes, mode, budget, comps, tiles)) > 0


def _ctypes_to_device(arr, nbytes, device):
    host = torch.frombuffer(bytearray(ctypes.string_at(ctypes.addressof(arr), nbytes)),
                            dtype=torch.uint8) if nbytes else torch.zeros(0, dtype=torch.uint8)
    dev = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=device)
    if nbytes:
        dev[:nbytes].copy_(host)
    return dev


def check_rows(a, n, device, what):
    """ValueError unless a is float64 [steps, max(n, 1), 4] on `device`: the kernels that get
    its address read or write all of it."""
    if not (torch.is_tensor(a) and a.dtype == torch.float64 and a.device == device and a.dim() == 3
            and tuple(a.shape[1:]) == (max(n, 1), 4)):
        raise ValueError('%s must be a float64 tensor [steps, %d, 4] on %s' % (what, max(n, 1), device))


def rows_contiguous(a):
    return len(a) == 0 or a[0].is_contiguous()


# SM time per pair of every compiled tile with three or more warps per scheduler (picoseconds;
# an ordered pair of the all-pairs modes, an unordered one of the others), from stage 1 at
# 65536 / 131072 bodies on GB300 (fp32un: the mean of a cube at rest and a Gaussian cloud).
TILE_COST = {
    'fp32': {(1, 128, 128): 73, (2, 128, 128): 70, (4, 128, 128): 70, (4, 128, 256): 69,
             (8, 128, 256): 72, (2, 256, 256): 66, (4, 256, 256): 69, (8, 256, 256): 69},
    'fp32n': {(1, 128, 128): 93, (2, 128, 128): 81, (4, 128, 128): 72, (4, 128, 256): 71,
              (8, 128, 256): 74, (4, 256, 256): 73},
    'fp32c': {(1, 128, 128): 108, (2, 128, 128): 100, (4, 128, 256): 98, (4, 256, 256): 95},
    'fp32u': {(4, 128, 128): 87, (4, 256, 256): 85, (8, 128, 256): 64, (4, 128, 256): 71,
              (2, 256, 256): 101, (8, 256, 256): 63, (8, 128, 128): 81, (8, 128, 64): 85,
              (4, 64, 64): 90, (8, 64, 64): 67, (16, 64, 64): 64},
    'fp32un': {(4, 128, 128): 98, (8, 128, 256): 74, (8, 128, 128): 74, (8, 128, 64): 78,
               (4, 128, 256): 79, (4, 256, 256): 75, (4, 64, 64): 103, (8, 64, 64): 77,
               (8, 64, 128): 75},
    'fp32cu': {(4, 128, 128): 114, (8, 128, 256): 57, (4, 128, 256): 61, (4, 256, 256): 88,
               (8, 128, 128): 86, (4, 64, 64): 118, (8, 64, 64): 88},
}


def tile_time(mode, tile, info, sm_count, resident):
    """Estimated step time (us) of a plan: the busiest SM's units at the tile's cost, slower
    where fewer than three warps per scheduler are resident (half the rate with one, 0.8 with
    two), plus the slots' traffic in stage 2 (24 bytes per entry, written and read, at ~8
    TB/s).  Over the unique-pair modes at 300-131072 bodies (56 measured sets of tiles) the
    tile it picks ran within 0.2 % of the fastest on average, at worst 7 % (fp32cu at 6500
    bodies, fp32un at 9000), over the all-pairs modes within 0.4 %; the rule before it, which
    did not count the CTAs that share an SM, was 5-30 % off above 8192 bodies."""
    grid = min(info.grid, info.n_units)
    on_sm = min(-(-grid // sm_count), resident)
    warps = on_sm * tile.threads / 128.0
    rate = (1.0 if warps >= 3 else 0.8 + 0.2 * (warps - 2) if warps >= 2 else
            0.5 + 0.3 * (warps - 1) if warps >= 1 else 0.5 * warps)
    cost = TILE_COST.get(mode, {}).get(tile.key(), 100.0)
    units = -(-info.n_units // grid) * on_sm
    return (units * info.itile * tile.jtile * cost * 1e-6 / rate +
            info.n_slots * info.itile * 24 / 8e6)


# Longest j-tile the default picks, and other shapes it may: FP32 partial sums run over one
# j-tile.  rms force error of fp32un at 8191 / 65536 bodies: 4/64/64 1.3e-7 / 5.6e-8, 8/64/64
# 1.5 / 7.5, 8/128/128 1.7 / 7.0, 8/64/128 1.7 / 8.0, 8/128/256 1.9 / 7.4.
DEFAULT_JTILE_MAX = {'fp32u': 64, 'fp32un': 64}
DEFAULT_ALSO = {'fp32un': [(8, 128, 128)]}
# And shapes it may pick where no CTA has more than one unit.  fp32un from 6145 to ~7300 bodies:
# 4/128/128 28.8-30.0 us a step (rms force error 1.4e-7 - 1.3e-7), 8/128/128 34.1-35.9 (1.3e-7 -
# 1.2e-7), 8/64/64 31.9-37.7, 4/64/64 29.0-37.9.
DEFAULT_ONE_WAVE = {'fp32un': [(4, 128, 128)]}


def default_tile(mode, sizes, device=None):
    """Tile shape used when no tuned entry exists: of the shapes with short partial sums
    (DEFAULT_JTILE_MAX, else 128 bodies) the one with the smallest estimated step time
    (tile_time)."""
    info = device_info(device)
    cands = fitting_tiles(sizes, mode) or tile_list(mode)
    longest = DEFAULT_JTILE_MAX.get(mode, 128)
    also = DEFAULT_ALSO.get(mode, ())
    one_wave = DEFAULT_ONE_WAVE.get(mode, ())
    cands = [t for t in cands if t.jtile <= longest or t.key() in also or t.key() in one_wave] or cands
    best = None
    for t in cands:
        occ = occupancy(mode, t, device)
        if occ <= 0:
            continue
        t.grid = info.sm_count * occ
        pinfo, _, _ = make_plan(sizes, 1.0, t, mode)
        if t.key() in one_wave and pinfo.n_units > t.grid:
            continue
        # no pairs at all (only empty universes): stage 1 launches nothing, any compiled
        # shape serves
        score = tile_time(mode, t, pinfo, info.sm_count, occ) if pinfo.n_units else float('inf')
        if best is None or score < best[0]:
            best = (score, t)
    if best is None:
        raise RuntimeError('no compiled tile shape fits mode %r' % (mode,))
    return best[1]


def fp64_pair_tile(sizes, sm_count, budget=None):
    """Tile of the FP64 unique-pair kernel for this workload, or None where its slots do not
    fit the slot budget (the ordered-pair kernel, with a few MB of them, then serves; slots
    take 24 bytes per body and row block before it: 0.7 GB at 60000 bodies, 34 GB at 600000;
    a GB300's budget ends at ~630000).  The time is the FP64
    instructions of the busiest SM: ceil(units / SMs) units of 32 columns against a block of
    32, 64 or 128 rows, 20 per pair, and three per column slot and row in stage 2; small
    blocks win where units are few (a step at 300 bodies: 12.5 us with 32 rows, 31 with 128;
    at 8191 1.24-1.26 ms with any), large ones keep the slots few."""
    if not any(sizes):
        return None
    best = None
    for rows in (32, 64, 128):
        t = _lib.Tile(1, rows, 32, sm_count)
        if not plan_fits(sizes, t, _lib.GRAV_MODE_FP64U, budget):
            continue
        info = make_plan(sizes, 1.0, t, _lib.GRAV_MODE_FP64U)[0]
        slots = sum(-(-n // rows) * n / 2 for n in sizes)
        cost = -(-info.n_units // sm_count) * rows * 20 + slots * 3 / 32 / sm_count
        if best is None or cost < best[0]:
            best = (cost, t)
    return best and best[1]


FUSED_MODES = ('fp32', 'fp32n', 'fp32c')
# (largest n, (threads, rows)) of the single-launch step, the fastest measured on GB300
# (graph-replayed steps of plain fp32, against the two-launch step's 7.6-8.3 us): n <= 32 --
# 3.5 us (one CTA); 64 -- 4.0 (one CTA); 128 -- 4.5 (a cluster of 4 CTAs); 256 -- 5.2 (8);
# 512 -- 5.9 (16).  From 1024 bodies the two-launch step, whose stage 1 spreads the pairs over
# every SM, is faster (8.4 us against 9.0).  fp32n and fp32c take grav_steps instead (1.9 us at
# 64 bodies, 3.6 at 1000) unless `fused` is given.
FUSED_RULE = ((32, (256, 64)), (64, (512, 64)), (128, (256, 32)), (512, (512, 32)))


def default_fused(mode, sizes, dev_info=None):
    """(threads, rows) of the single-launch step (grav_step_fused) for this workload, or
    None for the two-launch step: one universe of at most 512 bodies in an all-pairs
    FP32 mode."""
    if len(sizes) != 1 or mode not in FUSED_MODES:
        return None
    n = int(sizes[0])
    for n_max, cfg in FUSED_RULE:
        if 0 < n <= n_max:
            return cfg
    return None


# Largest universe whose queued steps (and accelerations alone) run as one launch
# (grav_steps), and up to which a single queued step does.  Measured on GB300, us per step of
# 20 queued / accelerations alone / one step, in brackets the two-launch step:
#   fp32n   64: 1.9 / 2.9 / 3.3 [8.5]   1000: 3.6 / 5.4 / 6.4 [9.1]   3000: 7.9 / 9.6 / 12.3 [13]
#           4096: 11.8 / 13.8 / 16.9 [17.7]   6000: 21.2 / 23 / 28 [33]   12000: 74 / 74 / 84 [105]
#   fp32c   1000: 3.6 / 5.5 / 6.5 [11.1]   4096: 14.0 / 16.4 / 19.5 [19.3]   6000: 25 / 28 / 33 [37]
# The unique-pair modes' own kernels pass it at 8000-9000 bodies (fp32un, default tile: 24 us
# against 35 at 6500, 36 against 37 at 8192, 51 against 51 at 10000), but their worst body is
# nearer there (force error of a cube / a Gaussian cloud at 8000 bodies, rows sharing their near
# radius: rms 1.2e-7 / 0.8e-7 in both, max 2.2e-6 / 3.5e-6 against 1.5e-6 / 1.8e-6), so they
# start at 6145.  fp32n has no such kernels: its ordered pairs in two launches are no nearer
# (9000 bodies: rms 1.9e-7 / 1.5e-7, here 1.8e-7 / 1.5e-7).  The plain modes, whose error is the
# rounding of the positions, keep their own kernels and their sums bit for bit.  After a single
# step the last CTA moves the positions over, which from ~2500 bodies on costs what the second
# launch does.
STEPS_MAX_N = {'fp32n': 12288, 'fp32c': 6144, 'fp32un': 6144, 'fp32cu': 6144}
STEPS_SINGLE_MAX_N = 2048


def default_steps(mode, sizes, dev_info):
    """True when the queued steps of this workload run as one launch (grav_steps): one
    universe within the measured size rule that the kernel takes on this GPU."""
    if len(sizes) != 1 or not 0 < sizes[0] <= STEPS_MAX_N.get(mode, 0):
        return False
    return bool(_lib.load().grav_steps_supported(_lib.MODES[mode], sizes[0], dev_info.sm_count))


class Engine:
    """Packed batch of universes on one GB300 with FP64 state.

    Parameters
      sizes : list of body counts (one per universe)
      T     : time step (scalar or one per universe)
      mode  : 'fp32' (default, all pairs), 'fp32u' (unique pairs), 'fp32n' / 'fp32un'
              (near pairs from double-single separations), 'fp32c' / 'fp32cu'
              (double-single separations for every pair) or 'fp64'
      tile  : _lib.Tile, or None to use the autotuner's choice / the default shape
      fused : single-launch step (grav_step_fused) for one small universe: (threads,
              rows) per CTA, False for the two-launch step, None to decide by size
              (default_fused, and default_steps: all queued steps in one launch)
    """

    def __init__(self, sizes, T, mode='fp32', tile=None, device=None, tuner=None, fused=None):
        self.lib = _lib.load()
        self.dev_info = device_info(device)
        self.device = torch.device('cuda', self.dev_info.index)
        if isinstance(mode, str):
            if mode not in _lib.MODES:
                raise ValueError('unknown precision mode %r (%s)' % (mode, ', '.join(_lib.MODES)))
            self.mode_name, self.mode = mode, _lib.MODES[mode]
        else:
            self.mode = int(mode)
            names = {v: k for k, v in _lib.MODES.items()}
            names[_lib.GRAV_MODE_FP64U] = 'fp64'
            self.mode_name = names[self.mode]
        self.sizes = [int(x) for x in sizes]
        self.T = list(T) if np.ndim(T) else [float(T)] * len(self.sizes)
        # queued steps in one launch, unless the caller picks the kernels himself
        self.chained = (fused is None and tile is None
                        and default_steps(self.mode_name, self.sizes, self.dev_info))
        if fused is None:
            fused = default_fused(self.mode_name, self.sizes, self.dev_info)
        if tile is None and self.mode == _lib.GRAV_MODE_FP64:
            tile = fp64_pair_tile(self.sizes, self.dev_info.sm_count,
                                  slot_budget_bytes(self.dev_info.index))
            if tile is not None:
                self.mode = _lib.GRAV_MODE_FP64U
                tile.grid = 0
        if tile is None:
            if tuner is not None and not fused and not self.chained:
                tile = tuner.choose(self.mode_name, self.sizes, self.dev_info, T=self.T)
            else:
                tile = default_tile(self.mode_name, self.sizes, self.dev_info.index)
        elif tile.grid <= 0:
            tile = _lib.Tile(tile.bpt, tile.threads, tile.jtile,
                             self.dev_info.sm_count * occupancy(self.mode, tile, self.dev_info.index))
        if not self.lib.grav_tile_supported(self.mode, ctypes.byref(tile)):
            raise ValueError('tile %r is not compiled for mode %s' % (tile, self.mode_name))
        self.tile = tile
        self.info, univ, seg = make_plan(self.sizes, self.T, tile, self.mode)
        info = self.info
        dev = self.device
        self.univ_dev = _ctypes_to_device(univ, ctypes.sizeof(_lib.UnivDesc) * info.n_univ, dev)
        self.seg_dev = _ctypes_to_device(seg, ctypes.sizeof(_lib.SegDesc) * info.n_seg, dev)
        self.univ_host = univ
        self.seg_host = seg
        nb = max(info.n_bodies, 1)
        self.r = torch.zeros((nb, 4), dtype=torch.float64, device=dev)
        self.v = torch.zeros((nb, 4), dtype=torch.float64, device=dev)
        self.a = torch.zeros((nb, 4), dtype=torch.float64, device=dev)
        pos_bytes = int(self.lib.grav_pos_bytes(self.mode, info.n_pad_total))
        self.pos = torch.zeros(max(pos_bytes // 4, 4), dtype=torch.float32, device=dev)
        part_bytes = int(self.lib.grav_part_bytes(ctypes.byref(info)))
        self.part = torch.zeros(max(part_bytes // 8, 1), dtype=torch.float64, device=dev)
        self.err = torch.zeros(1, dtype=torch.int32, device=dev)
        b = _lib.Batch()
        b.mode = self.mode
        b.n_univ = info.n_univ
        b.n_seg = info.n_seg
        b.n_slots = info.n_slots
        b.n_bodies = info.n_bodies
        b.n_pad_total = info.n_pad_total
        b.n_units = info.n_units
        b.tile = _lib.Tile(tile.bpt, tile.threads, tile.jtile, info.grid)
        b.eps2 = 1e-30
        b.univ = self.univ_dev.data_ptr()
        b.seg = self.seg_dev.data_ptr()
        b.r = self.r.data_ptr()
        b.v = self.v.data_ptr()
        b.pos = self.pos.data_ptr()
        b.part = self.part.data_ptr()
        b.a_out = self.a.data_ptr()
        b.err = self.err.data_ptr()
        self.batch = b
        self._bref = ctypes.byref(b)
        self.offsets = np.array([u.body_off for u in list(univ)[:info.n_univ]], dtype=np.int64)
        self.fused = None
        if fused:
            threads, rows = int(fused[0]), int(fused[1])
            n = self.sizes[0] if len(self.sizes) == 1 else -1
            if len(self.sizes) != 1 or not self.lib.grav_fused_supported(self.mode, n, threads, rows):
                raise ValueError('no single-launch step for mode %s, sizes %s, %d threads, %d rows'
                                 % (self.mode_name, self.sizes[:4], threads, rows))
            occ = ctypes.c_int32()
            with torch.cuda.device(dev):
                check(self.lib.grav_fused_occupancy(self.mode, n, threads, rows, ctypes.byref(occ)))
            if -(-n // rows) > occ.value * self.dev_info.sm_count:
                raise ValueError('%d CTAs of the single-launch step are not resident at once'
                                 % -(-n // rows))
            self.fused = (threads, rows)
            # grid-barrier counters of grav_step_fused (zero between calls)
            self.sync = torch.zeros(2, dtype=torch.int32, device=dev)
        self.scratch = None
        self._owes_stage1 = False
        if self.chained:
            # exchange buffers of grav_steps (zeroed once, then its own)
            nbytes = int(self.lib.grav_steps_scratch_bytes(self.sizes[0]))
            self.scratch = torch.zeros(nbytes, dtype=torch.uint8, device=dev)

    # ---- state ----------------------------------------------------------------------
    def set_state(self, r, v, gm, stream=None):
        """Load positions, velocities and G*m (already scaled) for all bodies, packed."""
        n = self.info.n_bodies
        if n and self.r.is_cuda and all(torch.is_tensor(x) and x.device == self.r.device
                                        for x in (r, v, gm)):
            self._load(r, v, gm, stream)
            return
        r = torch.as_tensor(np.asarray(r, dtype=np.float64).reshape(n, 3) if not torch.is_tensor(r)
                            else r.reshape(n, 3), dtype=torch.float64)
        v = torch.as_tensor(np.asarray(v, dtype=np.float64).reshape(n, 3) if not torch.is_tensor(v)
                            else v.reshape(n, 3), dtype=torch.float64)
        gm = torch.as_tensor(np.asarray(gm, dtype=np.float64).reshape(n) if not torch.is_tensor(gm)
                             else gm.reshape(n), dtype=torch.float64)
        if not bool(torch.isfinite(gm).all()) or bool((gm < 0).any()):
            raise ValueError('G*m must be finite and >= 0')
        max_gm = float(gm.max()) if n else 0.0
        self.batch.eps2 = float(self.lib.grav_eps2(max_gm))
        with torch.cuda.stream(self._stream(stream)):
            self.r[:n, :3].copy_(r, non_blocking=False)
            self.r[:n, 3].copy_(gm)
            self.v[:n, :3].copy_(v)
            self.v[:n, 3].zero_()
        self.prepare(stream)

    def _load(self, r, v, gm, stream):
        """set_state from tensors on the engine's device: two launches and one wait."""
        n = self.info.n_bodies
        r, v, gm = (x.detach().reshape(shape).to(torch.float64)
                    for x, shape in ((r, (n, 3)), (v, (n, 3)), (gm, (n,))))
        gm = gm.contiguous()
        span = torch.empty(2, dtype=torch.float64, device=self.r.device)
        check(self.lib.grav_gm_range(gm.data_ptr(), n, span.data_ptr(), self._h(None)))
        max_gm, bad = span.tolist()
        if bad:
            raise ValueError('G*m must be finite and >= 0')
        self.batch.eps2 = float(self.lib.grav_eps2(max_gm))
        if stream is not None:
            for x in (r, v, gm):
                x.record_stream(stream)
            # r and v may be `stream`'s own work: strided ones are packed there
            with torch.cuda.stream(stream):
                r, v = r.contiguous(), v.contiguous()
        else:
            r, v = r.contiguous(), v.contiguous()
        check(self.lib.grav_load_state(r.data_ptr(), v.data_ptr(), gm.data_ptr(), n,
                                       self.r.data_ptr(), self.v.data_ptr(), self._h(stream)))
        self.prepare(stream)

    def generate_state(self, scenarios, G, stream=None):
        """Fill r and v on the device from seeded scenarios (gravitation_gb300.generate):
        one list of parts per universe, covering exactly that universe's bodies; G is
        the (scaled) constant the G*m column is formed with (one per universe or one
        for all).  Sets eps2 from the largest G*m and refreshes the stage-1 positions."""
        from . import generate as gen
        if len(scenarios) != len(self.sizes):
            raise ValueError('%d scenarios for %d universes' % (len(scenarios), len(self.sizes)))
        Gs = list(G) if np.ndim(G) else [float(G)] * len(self.sizes)
        st = self._stream(stream)
        for u, parts in enumerate(scenarios):
            n = self.sizes[u]
            if gen.total_bodies(parts) != n or sum(p.n for p in parts) != n:
                raise ValueError('scenario of universe %d does not cover its %d bodies' % (u, n))
            o = int(self.offsets[u])
            gen.generate(parts, self.r[o:o + n], self.v[o:o + n], Gs[u], st)
        nb = self.info.n_bodies
        st.synchronize()  # r may be host memory the device wrote (bind_host_state)
        with torch.cuda.stream(st):
            max_gm = float(self.r[:nb, 3].max()) if nb else 0.0
        self.batch.eps2 = float(self.lib.grav_eps2(max_gm))
        self.prepare(st)

    def bind_host_state(self, hr, hv):
        """Keep r and v in page-locked host tensors hr, hv (float64 [n_bodies, 4], same
        layout): prepare and stage 2 then read and write them in place over the CPU-GPU
        link, and the device copies are no longer used.  Returns False, changing
        nothing, if the tensors are not page-locked memory the device can address."""
        n = self.info.n_bodies
        for t in (hr, hv):
            if (t.device.type != 'cpu' or t.dtype != torch.float64 or tuple(t.shape) != (n, 4)
                    or not t.is_contiguous()):
                raise ValueError('host state must be contiguous float64 [%d, 4] CPU tensors' % n)
        ptrs = []
        for t in (hr, hv):
            p = ctypes.c_void_p()
            if not t.is_pinned() or self.lib.grav_host_device_pointer(
                    ctypes.c_void_p(t.data_ptr()), ctypes.byref(p)) != _lib.GRAV_OK:
                return False
            ptrs.append(p.value)
        self.r, self.v = hr, hv
        self.batch.r, self.batch.v = ptrs
        return True

    def _stream(self, stream):
        return stream if stream is not None else torch.cuda.current_stream(self.device)

    def _h(self, stream):
        return ctypes.c_void_p(self._stream(stream).cuda_stream)

    # ---- stages ---------------------------------------------------------------------
    def prepare(self, stream=None):
        """Refresh the padded stage-1 positions after r was changed."""
        check(self.lib.grav_prepare(self._bref, self._h(stream)))

    def stage1(self, stream=None):
        self._owes_stage1 = False
        check(self.lib.grav_stage1(self._bref, self._h(stream)))

    def stage2(self, flags=_lib.GRAV_S2_INTEGRATE, stream=None):
        """Stage 2 over the partial sums that stage 1, or forces(), left (queued steps in one
        launch leave none)."""
        if self._owes_stage1:
            self.stage1(stream)
        check(self.lib.grav_stage2(self._bref, int(flags), self._h(stream)))

    def step(self, steps=1, stream=None, write_a=False):
        """`steps` full steps (stage 1 + stage 2, the single-launch step, or all of them in
        one launch) queued on the stream."""
        flags = _lib.GRAV_S2_INTEGRATE | (_lib.GRAV_S2_WRITE_A if write_a else 0)
        h = self._h(stream)
        self._owes_stage1 = False
        if self.chained and (int(steps) > 1 or int(steps) == 1 and self.sizes[0] <= STEPS_SINGLE_MAX_N):
            self._steps(flags, int(steps), 0, h)
            return
        if self.fused:
            threads, rows = self.fused
            sync = ctypes.c_void_p(self.sync.data_ptr())
            for _ in range(int(steps)):
                check(self.lib.grav_step_fused(self._bref, flags, threads, rows, sync, h))
            return
        for _ in range(int(steps)):
            check(self.lib.grav_step(self._bref, flags, h))

    def _steps(self, flags, steps, a_stride, h):
        check(self.lib.grav_steps(self._bref, flags, steps, a_stride,
                                  ctypes.c_void_p(self.scratch.data_ptr()), h))

    def steps_to(self, a, stream=None):
        """len(a) full steps, step k's accelerations written to a[k] (float64
        [steps, n_bodies, 4], device; each a[k] contiguous, and apart from the others)."""
        check_rows(a, self.info.n_bodies, self.device, 'a')
        if not rows_contiguous(a) or len(a) > 1 and a.stride(0) < a[0].numel():
            raise ValueError('the rows of each step must be contiguous and the steps apart')
        if not len(a):
            return
        flags = _lib.GRAV_S2_INTEGRATE | _lib.GRAV_S2_WRITE_A
        h = self._h(stream)
        keep = self.batch.a_out
        try:
            if self.chained:
                self.batch.a_out = a.data_ptr()
                self._steps(flags, len(a), a.stride(0), h)
                return
            for k in range(len(a)):
                self.batch.a_out = a[k].data_ptr()
                check(self.lib.grav_step(self._bref, flags, h))
        finally:
            self.batch.a_out = keep

    def capture_graph(self, steps=1):
        """CUDA graph of `steps` full steps (one launch, or stage 1 + stage 2: 2 launches
        per step); returns a torch.cuda.CUDAGraph whose replay() runs them.  It holds the
        eps2 of the masses loaded: capture again after set_state with other masses.
        The launches are recorded on a side stream that torch puts into capture mode."""
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream(self.device))
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            self.step(steps, stream=side)
        torch.cuda.current_stream(self.device).wait_stream(side)
        return g

    def forces(self, stream=None):
        """Stage 1 only; returns the accelerations (float64 [n_bodies, 3], device)."""
        if self.chained:
            self._steps(_lib.GRAV_S2_WRITE_A, 1, 0, self._h(stream))
            self._owes_stage1 = True   # should stage2 follow: this launch leaves no slots
            return self.a[:self.info.n_bodies, :3]
        self.stage1(stream)
        self.stage2(_lib.GRAV_S2_WRITE_A, stream)
        return self.a[:self.info.n_bodies, :3]

    # ---- diagnostics ----------------------------------------------------------------
    DIAG_TILE = (2, 128, 128)

    def _fp64_view(self):
        """An FP64-mode batch sharing r and v, with its own all-pairs plan, padded double4
        positions and partial-sum scratch (so a diagnostic never clobbers stage 1)."""
        if getattr(self, '_b64', None) is None:
            t = _lib.Tile(*self.DIAG_TILE, 0)
            t.grid = self.dev_info.sm_count * max(
                occupancy(_lib.GRAV_MODE_FP64, t, self.dev_info.index), 1)
            info, univ, seg = make_plan(self.sizes, self.T, t, 'fp64')
            dev = self.device
            self._univ64 = _ctypes_to_device(univ, ctypes.sizeof(_lib.UnivDesc) * info.n_univ, dev)
            self._seg64 = _ctypes_to_device(seg, ctypes.sizeof(_lib.SegDesc) * info.n_seg, dev)
            nbytes = int(self.lib.grav_pos_bytes(_lib.GRAV_MODE_FP64, info.n_pad_total))
            self._pos64 = torch.zeros(max(nbytes // 8, 4), dtype=torch.float64, device=dev)
            self._part64 = torch.zeros(max(int(self.lib.grav_part_bytes(ctypes.byref(info))) // 8,
                                           1), dtype=torch.float64, device=dev)
            self._out64 = torch.zeros(max(info.n_univ, 1) * 8, dtype=torch.float64, device=dev)
            b = _lib.Batch()
            b.mode = _lib.GRAV_MODE_FP64
            b.n_univ, b.n_seg, b.n_slots = info.n_univ, info.n_seg, info.n_slots
            b.n_bodies, b.n_pad_total, b.n_units = info.n_bodies, info.n_pad_total, info.n_units
            b.tile = _lib.Tile(t.bpt, t.threads, t.jtile, info.grid)
            b.eps2 = 1e-30
            b.univ, b.seg = self._univ64.data_ptr(), self._seg64.data_ptr()
            b.r, b.v = self.r.data_ptr(), self.v.data_ptr()
            b.pos, b.part = self._pos64.data_ptr(), self._part64.data_ptr()
            b.a_out, b.err = self.a.data_ptr(), self.err.data_ptr()
            self._b64 = b
        return self._b64

    def energy(self, G, stream=None):
        """FP64 (kinetic, potential, momentum[3]) per universe as a numpy array
        [n_univ, 5]; G is the (scaled) gravitational constant of the universes."""
        b = self._fp64_view()
        h = self._h(stream)
        check(self.lib.grav_prepare(ctypes.byref(b), h))
        check(self.lib.grav_energy(ctypes.byref(b), ctypes.c_void_p(self._out64.data_ptr()), h))
        out = self._out64.view(-1, 8)[:self.info.n_univ, :5].cpu().numpy() / float(G)
        self.raise_on_device_error()
        return out

    # ---- errors ---------------------------------------------------------------------
    def device_error(self):
        """Device error flag (GRAV_DEV_*); synchronises the stream."""
        return int(self.err.item())

    def raise_on_device_error(self):
        code = self.device_error()
        if code != _lib.GRAV_DEV_OK:
            self.err.zero_()
            raise _lib.GravError(_lib.GRAV_E_CUDA, 'device error flag %d (%s)' % (
                code, 'bounded wait expired: a bulk copy or a grid barrier'
                if code == _lib.GRAV_DEV_TIMEOUT else 'unknown'))

    # ---- views ----------------------------------------------------------------------
    def universe_slice(self, u):
        o = int(self.offsets[u])
        return slice(o, o + self.sizes[u])

    def interactions_per_step(self):
        """Algorithmic interactions per step: sum over universes of N^2."""
        return sum(n * n for n in self.sizes)
