"""Launch-configuration autotuner for the fused step.

The step is compiled in several launch configurations (block shape x register
budget, SW_STEP_CONFIGS in csrc/sw_step.cuh).  Which one hides memory latency
best depends on the storage type and the grid, so it is measured: each
configuration steps the solver's current state into its spare lattice a few
times (the state itself is not modified, and the spare lattice is overwritten
by the next real step anyway), timed with CUDA events, and the fastest is
installed for that storage type with sw_set_step_config.  Results are cached
per (device name, dtype, grid, alone) for the life of the process.

A timing decides between configurations that give the same bits, and between no
others: what a solve computes must not depend on which of two close times came
out smaller.  The 16-bit types have two families of them -- one cell per thread
(0-3) and two (4 and up), whose packed arithmetic rounds differently -- and the
size of the wall decides which of them the tuner chooses among (candidates).
"""
import torch

from . import _native as N
from .fields import _stream
from .lattice import Q

_CACHE = {}


def config_count():
    return N.lib().sw_step_config_count()


def one_cell_sums(grid):
    """Whether accumulating steps of a 16-bit wall of this grid run one cell per thread.  They do from
    where the two-cell blocks (64 cells of 4 rows) need a second wave on the 152 SMs, eight to each,
    which the shorter blocks fill better, up to where lattices, sums and flags leave the L2 and the
    wider accesses win (captured graphs, us per step, one cell / two: 1080 blocks 10.03 / 9.52, 1216
    10.11 / 10.83, 1230 10.43 / 10.11, 1360 10.33 / 10.82, 2040 11.9 / 14.2, 3000 15.0 / 18.3; 93 MB
    21.1 / 21.8, 105 MB 25.35 / 25.17, 126 MB 33.8 / 30.3, 143 MB 39.1 / 32.5)."""
    blocks = (grid.pitch // 32 + 1) // 2 * ((grid.ny + 3) // 4) * grid.nz
    return blocks >= 8 * 152 and grid.cells_padded * (2 * Q * 2 + 4 * 8 + 1) < 110e6


def candidates(dtype, grid=None, accumulating=False):
    """The configurations that tuning may install for a storage type: all give the same bits.
    16 bits: two cells per thread, or one for the accumulating steps of some grids (one_cell_sums).
    Plain steps are the fastest with two at every size measured (captured graphs, fp16, us per step,
    best of 0-3 / best of 4-17: H 8 9.1 / 7.1, H 12 11.1 / 9.8, H 16 21.6 / 17.7, H 24 77.1 / 62.7)."""
    if dtype not in (N.SW_F16_SHIFT, N.SW_BF16_SHIFT):
        return range(config_count())
    if grid is not None and accumulating and one_cell_sums(grid):
        return range(4)
    return range(4, config_count())


def time_configs(solver, repeats=8, warmup=2, acc=None, cfgs=None):
    """Mean step time in ms of every configuration (or of `cfgs`) on the solver's grid (with `acc`,
    an Accum that receives throw-away sums, the accumulating variant).  A configuration whose TMA-staged
    blocks gave up waiting for their copies (a time-out in its status word or in
    sw_tma_timeouts) computed an invalid step and is left out, so it can never win by skipping work."""
    from .fields import StatusWord
    L = N.lib()
    g = solver.grid
    src, dst = solver.f[solver.cur], solver.f[1 - solver.cur]
    stream = torch.cuda.current_stream()
    accp = acc.ptr if acc is not None else None
    status = StatusWord(device=solver.device)
    res = {}
    for cfg in range(config_count()) if cfgs is None else cfgs:
        status.clear()
        L.sw_tma_timeouts()                           # read and clear the process-wide counter

        def launch():
            return L.sw_step_checked(g.gp, src.dtype, src.ptr, dst.ptr, solver.flags.ptr, solver.flags.tiles_ptr,
                                     solver.uin.ptr, solver.nu0, solver.cs, solver.x_sponge, solver.nu_sponge,
                                     None, 0, accp, cfg, status.ptr, _stream(stream))
        rc = launch()
        if rc == N.SW_ERR_UNSUPPORTED:
            continue                                  # not compiled for this storage type
        N.check(rc, "sw_step_checked")
        for _ in range(warmup - 1):
            N.check(launch(), "sw_step_checked")
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(repeats):
            N.check(launch(), "sw_step_checked")
        e1.record()
        torch.cuda.synchronize()
        timed_out = bool(status.read() & N.SW_STATUS_TIMEOUT)
        if L.sw_tma_timeouts() != 0 or timed_out:      # (reading the counter also clears it)
            continue
        res[cfg] = e0.elapsed_time(e1) / repeats
    if not res:
        raise RuntimeError("no launch configuration completed a step without a device wait time-out")
    return res


def tune(solver, repeats=8, force=False, accumulating=True, alone=True):
    """Pick and install the fastest of the candidates for the solver's storage type, for plain and for
    accumulating steps; returns (cfg, times) of the plain steps.  alone=False: for walls of any size
    that share what is installed, whose bits must not follow the size of the one that is timed."""
    from .fields import Accum
    g = solver.grid
    key = (torch.cuda.get_device_name(solver.device), solver.dtype, g.nx, g.ny, g.nz, alone)
    if key in _CACHE and not force:
        best, times, best_acc = _CACHE[key]
    else:
        times = time_configs(solver, repeats=repeats, cfgs=candidates(solver.dtype))
        best = min(times, key=times.get)
        best_acc = best
        if accumulating:
            scratch = Accum(g, device=solver.device)
            acc_times = time_configs(solver, repeats=max(2, repeats // 2), acc=scratch,
                                     cfgs=candidates(solver.dtype, g if alone else None, accumulating=True))
            best_acc = min(acc_times, key=acc_times.get)
            del scratch
        _CACHE[key] = (best, times, best_acc)
    N.check(N.lib().sw_set_step_config(solver.dtype, best), "sw_set_step_config")
    N.check(N.lib().sw_set_step_config_accum(solver.dtype, best_acc), "sw_set_step_config_accum")
    return best, times


def current(dtype):
    return N.lib().sw_get_step_config(N.dtype_code(dtype))


__all__ = ["tune", "time_configs", "candidates", "one_cell_sums", "config_count", "current"]
