"""slc_trace_gather_bdf2_staged (gather source boxes staged in shared memory
by TMA) against slc_trace_gather_bdf2 (gather through L1): equal clamp counts
and bit-identical outputs, with every box staged (small dt), with many blocks
falling back to L1 (wide feet), and on a grid too shallow for a box.
The arithmetic of both is written with explicit roundings, so this holds at
both orders and whatever ptxas would otherwise fuse."""

import ctypes
import math

import pytest
import torch

from slchannel_b200 import _native as N
from slchannel_b200.fields import synthetic_channel_field
from slchannel_b200.solver import SLChannelFlow
from slchannel_b200.utils import compute_bulk_velocity

pytestmark = pytest.mark.gpu


def _flow(n3, dt, urms, order=6, traj=2, iters=2):
    nx, ny, nz = n3
    cfg = {"grid": {"nx": nx, "ny": ny, "nz": nz},
           "domain": {"Lx": 2 * math.pi, "Ly": math.pi, "Lz": 2.0},
           "flow": {"Re": 2800.0, "Re_tau": 180.0, "U_bulk": 1.0, "gamma": 2.0},
           "initialization": {"type": "parabolic"}, "time": {"dt": dt},
           "compute": {"device": "cuda"},
           "sl": {"interp_order": order, "traj_interp_order": traj, "n_traj_iters": iters, "interp_dtype": "fp64"}}
    f = SLChannelFlow(config=cfg)
    u, v, w = synthetic_channel_field(nx, ny, nz, 2 * math.pi, math.pi, 2.0, f.z_f.cpu().numpy(),
                                      f.z_c.cpu().numpy(), urms=urms, seed=3)
    f.set_state(*(torch.from_numpy(a) for a in (u, v, w)))
    f.apply_bc_uvw()
    f.u *= 1.0 / float(compute_bulk_velocity(f.u, f.cell_vol_ratio, f.total_volume))
    f._save_and_project_initial()
    for _ in range(2):
        f.step_sl_bdf2(dt)
    return f


def _both(f, dt):
    cur, prev = (f.u, f.v, f.w), (f.u_nm1, f.v_nm1, f.w_nm1)
    res = []
    for name in ("slc_trace_gather_bdf2", "slc_trace_gather_bdf2_staged"):
        out = [torch.zeros_like(t) for t in cur]
        ncl = torch.zeros((), dtype=torch.int64, device=f.device)
        f._grid.call(name, *[N.ptr(t) for t in cur], *[N.ptr(t) for t in prev], float(dt),
                     *[N.ptr(t) for t in out], N.ptr(ncl), N.stream_of(f.u))
        res.append((out, int(ncl)))
    torch.cuda.synchronize()
    stats = (ctypes.c_int64 * 4)()
    N.lib().slc_gather_stats(f._grid.handle, stats, 1)
    return res, list(stats)


@pytest.mark.parametrize("order", [6, 4])
def test_staged_equals_l1_all_staged(order):
    f = _flow((40, 24, 48), 0.01, 0.1, order)
    (a, na), (b, nb) = _both(f, 0.01)[0]
    for c, x, y in zip("uvw", a, b):
        assert torch.equal(x, y), c
    assert na == nb
    stats = _both(f, 0.01)[1]
    assert stats[0] == 0 and stats[1] > 0 and stats[2] == stats[1] and stats[3] == stats[1]


def test_staged_equals_l1_wide_feet():
    f = _flow((24, 16, 48), 0.6, 0.35)
    (a, na), (b, nb) = _both(f, 0.6)[0]
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    assert na == nb and na > 0
    stats = _both(f, 0.6)[1]
    assert stats[0] == 0 and stats[3] < stats[1]  # some blocks gathered through L1


def test_staged_on_a_shallow_grid_is_the_l1_path():
    f = _flow((20, 16, 24), 0.05, 0.1)
    (a, na), (b, nb) = _both(f, 0.05)[0]
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    assert na == nb
    assert _both(f, 0.05)[1][1] == 0


@pytest.mark.parametrize("order", [6, 4])
@pytest.mark.parametrize("axis", [0, 1])
def test_staged_equals_l1_thousands_of_cells_away(axis, order):
    """A uniform U* moving every foot by 5000.37 cells, so that all of a block's
    feet lie beyond the range the box search tells apart: V^n = U0 + a and
    V^{n-1} = U0 + 2 a with a random a."""
    f = _flow((64, 32, 40), 0.01, 0.1, order)
    g = torch.Generator().manual_seed(4)
    a = [0.1 * torch.randn(t.shape, generator=g, dtype=torch.float64).to(t.device) for t in (f.u, f.v, f.w)]
    cells, step = 5000.37, (f.dx, f.dy)[axis]
    for scale in (2.0, 1.0):  # V^{n-1}, then V^n
        for c, (t, r) in enumerate(zip((f.u, f.v, f.w), a)):
            t.copy_(scale * r)
            if c == axis:
                t += 1.0
            if c == 2:  # no flow through the walls
                t[:, :, 0] = 0.0
                t[:, :, -1] = 0.0
        f.apply_bc_uvw()
        if scale == 2.0:
            prev = [t.clone() for t in (f.u, f.v, f.w)]
    for t, p in zip((f.u_nm1, f.v_nm1, f.w_nm1), prev):
        t.copy_(p)
    (x, nx), (y, ny) = _both(f, cells * step)[0]
    for c, p, q in zip("uvw", x, y):
        assert torch.isfinite(p).all() and torch.equal(p, q), c
    assert nx == ny


@pytest.mark.parametrize("n3", [(40, 24, 48), (64, 20, 24)])
@pytest.mark.parametrize("order,traj,iters", [(6, 4, 2), (6, 4, 3), (6, 2, 3), (4, 4, 2), (4, 2, 1)])
def test_staged_equals_l1_other_trajectories(n3, order, traj, iters):
    """Tricubic trajectories and other iteration counts, near and spread feet."""
    for dt, urms in ((0.01, 0.1), (0.3, 0.35)):
        f = _flow(n3, dt, urms, order, traj, iters)
        (a, na), (b, nb) = _both(f, dt)[0]
        for c, x, y in zip("uvw", a, b):
            assert torch.isfinite(x).all() and torch.equal(x, y), (c, dt)
        assert na == nb


@pytest.mark.parametrize("nz", [31, 32, 33, 63, 64, 65, 96, 97, 129])
@pytest.mark.parametrize("order", [6, 4])
def test_staged_equals_l1_at_tile_edges(nz, order):
    """k_sl's 64- and 32-level tiles and the boxes' four levels against each other
    around the tiles' ends (w has one level fewer)."""
    f = _flow((32, 10, nz), 0.03, 0.1, order)
    (a, na), (b, nb) = _both(f, 0.03)[0]
    for c, x, y in zip("uvw", a, b):
        assert float(x.abs().max()) > 0.0 and torch.equal(x, y), c
    assert na == nb
