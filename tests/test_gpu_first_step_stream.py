"""A new handle's first step on a stream that does not wait for the default one:
what the handle clears or uploads when it is made or first used must be done, or
ordered before, wherever that work goes.  Steps from a handle's creation on an
idle side stream must equal those on the default stream bit for bit."""

import math

import pytest
import torch

from slchannel_b200.fields import synthetic_channel_field
from slchannel_b200.host import HostStateStepper, pinned_like
from slchannel_b200.solver import SLChannelFlow
from slchannel_b200.utils import generate_grid

pytestmark = pytest.mark.gpu

NX, NY, NZ, DT = 96, 80, 64, 0.02


def _flow(order, precision):
    return SLChannelFlow(config={
        "grid": {"nx": NX, "ny": NY, "nz": NZ},
        "domain": {"Lx": 2 * math.pi, "Ly": math.pi, "Lz": 2.0},
        "flow": {"Re": 2800.0, "Re_tau": 180.0, "U_bulk": 1.0, "gamma": 2.0},
        "initialization": {"type": "parabolic"}, "time": {"dt": DT}, "compute": {"device": "cuda"},
        "sl": {"interp_order": order, "n_traj_iters": 2, "interp_dtype": precision}})


def _fields():
    z_f, z_c, _, _ = (t.numpy() for t in generate_grid(2.0, NZ, 2.0))
    f = synthetic_channel_field(NX, NY, NZ, 2 * math.pi, math.pi, 2.0, z_f, z_c, urms=0.1, seed=2)
    return [torch.from_numpy(a).cuda() for a in f]


@pytest.mark.parametrize("order,precision", [(4, "fp64"), (6, "fp64"), (4, "mixed"), (6, "mixed")])
def test_first_step_on_a_side_stream(order, precision):
    V = _fields()
    got = []
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            f = _flow(order, precision)
            f.set_state(*V)
            for _ in range(2):  # BDF1, then the first BDF2
                bulk = f.step_sl_bdf2(DT)
        torch.cuda.synchronize()
        got.append([t.clone() for t in (f.u, f.v, f.w, f.p, *bulk)])
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_first_host_step_on_a_side_stream():
    V = _fields()
    got = []
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        f = _flow(6, "fp64")
        f.set_state(*V)
        f.step_sl_bdf2(DT)
        prev = [pinned_like(t).copy_(t) for t in (f.u_nm1, f.v_nm1, f.w_nm1)]
        cur = [pinned_like(t).copy_(t) for t in (f.u, f.v, f.w)]
        nxt = [pinned_like(t).fill_(7.0) for t in cur]
        p, bulk = pinned_like(f.p).fill_(7.0), torch.zeros(2, dtype=torch.float64).pin_memory()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            HostStateStepper(f).step(cur, prev, nxt, p, bulk, DT)
        torch.cuda.synchronize()
        got.append([t.clone() for t in (*nxt, p, bulk)])
    for a, b in zip(*got):
        assert torch.equal(a, b)
