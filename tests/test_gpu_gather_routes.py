"""Which trace+gather an FP64 triquintic step takes, and that all give one result.

The step runs with x along the lanes where nx fills enough of them (from boxes,
or through L1 where the feet spread), else k_sl.  Routes are read off the
staged-box counters, which only the box kernel advances.  Every route has the
same arithmetic, so the step must equal its own pieces with k_sl as the
trace+gather (slc_trace_gather_bdf2, slc_zsolve, slc_project) bit for bit."""

import ctypes
import math

import pytest
import torch

from slchannel_b200 import _native as N
from slchannel_b200.ensemble import ChannelEnsemble
from slchannel_b200.fields import synthetic_channel_field
from slchannel_b200.solver import SLChannelFlow
from slchannel_b200.utils import compute_bulk_velocity

pytestmark = pytest.mark.gpu


def _flow(n3, dt, urms=0.1, order=6, traj=2, iters=2, direction=1.0):
    nx, ny, nz = n3
    f = SLChannelFlow(config={
        "grid": {"nx": nx, "ny": ny, "nz": nz},
        "domain": {"Lx": 2 * math.pi, "Ly": math.pi, "Lz": 2.0},
        "flow": {"Re": 2800.0, "Re_tau": 180.0, "U_bulk": direction, "gamma": 2.0},
        "initialization": {"type": "parabolic"}, "time": {"dt": dt}, "compute": {"device": "cuda"},
        "sl": {"interp_order": order, "traj_interp_order": traj, "n_traj_iters": iters, "interp_dtype": "fp64"}})
    u, v, w = synthetic_channel_field(nx, ny, nz, 2 * math.pi, math.pi, 2.0, f.z_f.cpu().numpy(),
                                      f.z_c.cpu().numpy(), urms=urms, seed=3)
    f.set_state(*(torch.from_numpy(a) for a in (u, v, w)))
    f.apply_bc_uvw()
    f.u *= direction / float(compute_bulk_velocity(f.u, f.cell_vol_ratio, f.total_volume))
    f._save_and_project_initial()
    f.step_sl_bdf2(dt)  # bootstrap
    return f


def _blocks(handle):
    s = (ctypes.c_int64 * 4)()
    N.check(N.lib().slc_gather_stats(handle, s, 0), handle)
    assert s[0] == 0
    return s[1]


@pytest.mark.parametrize("n3,traj,boxes", [
    ((24, 16, 48), 2, True),     # less than a wave of blocks
    ((24, 96, 64), 2, False),    # a quarter of the lanes idle, copies three times the grid
    ((32, 64, 24), 2, True),
    ((33, 40, 64), 2, False),    # half of the lanes idle
    ((48, 40, 48), 2, True),     # three quarters in use
    ((16, 64, 64), 2, False),
    ((64, 20, 24), 4, True),     # tricubic trajectories: full lanes, shallow or wide
    ((48, 40, 48), 4, False),
    ((64, 16, 100), 4, False),
    ((96, 12, 100), 4, True),
])
def test_route(n3, traj, boxes):
    f = _flow(n3, 0.01, traj=traj)
    f.step_sl_bdf2(0.01)
    torch.cuda.synchronize()
    assert (_blocks(f._grid.handle) > 0) == boxes


def _pieces_equal_the_step(f, dt):
    cur, prev = [f.u, f.v, f.w], [f.u_nm1, f.v_nm1, f.w_nm1]
    got = []
    for whole in (True, False):
        out = [torch.zeros_like(t) for t in cur]
        p = torch.zeros_like(f.p)
        ncl = torch.zeros((), dtype=torch.int64, device=f.device)
        if whole:
            (pc, k1), (pp, k2), (pn, k3) = (N.ptr_array(t) for t in (cur, prev, out))
            f._grid.call("slc_step_bdf2", pc, pp, pn, N.ptr(p), float(dt), N.ptr(ncl), N.stream_of(p))
        else:
            f._grid.call("slc_trace_gather_bdf2", *[N.ptr(t) for t in cur], *[N.ptr(t) for t in prev], float(dt),
                         *[N.ptr(t) for t in out], N.ptr(ncl), N.stream_of(p))
            dt_eff = (2.0 / 3.0) * dt
            f._grid.call("slc_zsolve", *[N.ptr(t) for t in out], dt_eff, N.stream_of(p))
            f._grid.call("slc_project", *[N.ptr(t) for t in out], N.ptr(p), dt_eff, dt_eff, N.stream_of(p))
        torch.cuda.synchronize()
        got.append((*out, p, ncl))
    for a, b in zip(*got):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("n3", [(61, 18, 23), (64, 16, 100), (94, 14, 11), (97, 10, 36)])
@pytest.mark.parametrize("traj,iters", [(2, 2), (2, 1), (2, 3), (4, 2), (4, 3)])
@pytest.mark.parametrize("wide", [False, True])
def test_step_equals_its_pieces_with_k_sl(n3, traj, iters, wide):
    dt = 0.6 if wide else 0.01
    f = _flow(n3, dt, 0.35 if wide else 0.1, traj=traj, iters=iters)
    for _ in range(3):  # the choice between boxes and L1 has settled
        f.step_sl_bdf2(dt)
        torch.cuda.synchronize()
    before = _blocks(f._grid.handle)
    _pieces_equal_the_step(f, dt)
    if wide:
        assert _blocks(f._grid.handle) == before  # the feet spread: not from boxes


@pytest.mark.parametrize("n3,traj,dt", [((72, 64, 128), 2, 0.02), ((96, 64, 96), 2, 0.2), ((72, 64, 128), 2, 0.25), ((80, 128, 64), 4, 0.02)])
def test_ensemble_of_large_instances_equals_its_channels(n3, traj, dt):
    """Instances with their own trace+gather launches: boxes, x along the lanes
    through L1, k_sl (nx leaves lanes idle and the feet spread, or the
    trajectories are tricubic)."""
    flows = [_flow(n, dt, traj=traj) for n in (n3, (16, 12, 20))]
    ens = ChannelEnsemble([_flow(n, dt, traj=traj) for n in (n3, (16, 12, 20))], [dt, dt], autotune=False)
    for _ in range(2):
        ens.step()
        for f in flows:
            f.step_sl_bdf2(dt)
    torch.cuda.synchronize()
    for i, f in enumerate(flows):
        for a, b in zip((*ens.velocity(i), ens.p[i]), (f.u, f.v, f.w, f.p)):
            assert float((a - b).abs().max()) <= 1e-12 * max(1.0, float(b.abs().max()))


@pytest.mark.parametrize("direction", [1.0, -1.0])
def test_ensemble_leaves_the_boxes_for_fast_mean_flow_either_way(direction):
    """At 1.5 cells of mean displacement a step a large instance gathers through
    L1, whichever way its flow goes."""
    for dt, boxes in ((0.05, True), (0.2, False)):  # 0.76 and 3.06 cells
        f = _flow((96, 64, 96), dt, direction=direction)
        ens = ChannelEnsemble([f], [dt], autotune=False)
        ens.step()
        torch.cuda.synchronize()
        handle = ctypes.c_void_p(N.lib().slc_ensemble_grid(ens._h, 0))
        assert (_blocks(handle) > 0) == boxes


def test_step_without_memory_for_the_copies():
    """Where the padded copies do not fit, the step runs k_sl instead of failing."""
    n3, dt = (96, 64, 40), 0.01
    fits, starved = _flow(n3, dt), _flow(n3, dt)
    fits.step_sl_bdf2(dt)  # boxes
    for f in (fits, starved):  # U* and the kernels
        out = [torch.zeros_like(t) for t in (f.u, f.v, f.w)]
        if f.u_nm1 is not None:
            f._grid.call("slc_trace_gather_bdf2", *[N.ptr(t) for t in (f.u, f.v, f.w, f.u_nm1, f.v_nm1, f.w_nm1)],
                         dt, *[N.ptr(t) for t in out], None, N.stream_of(f.u))
    starved._next = starved._alloc_next()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    copies = 6 * 8 * (96 + 48) * (64 + 10) * 40
    filler = torch.empty(torch.cuda.mem_get_info()[0] - copies // 2, dtype=torch.uint8, device="cuda")
    try:
        starved.step_sl_bdf2(dt)
        torch.cuda.synchronize()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert _blocks(starved._grid.handle) == 0 and _blocks(fits._grid.handle) > 0
    for a, b in zip((fits.u, fits.v, fits.w, fits.p), (starved.u, starved.v, starved.w, starved.p)):
        assert torch.equal(a, b)
