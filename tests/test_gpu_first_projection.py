"""The Poisson solve's inverse pivots are made at a handle's first projection:
making a handle launches nothing, and a first projection that a CUDA graph
captures gives the same result at every replay as one that runs at once."""

import math

import pytest
import torch

from slchannel_b200 import _native as N
from slchannel_b200.semilag import SLAdvector
from slchannel_b200.utils import generate_grid

pytestmark = pytest.mark.gpu

NX, NY, NZ, LX, LY, LZ = 20, 18, 13, 2 * math.pi, math.pi, 2.0


def _advector():
    z_f, z_c, _, _ = generate_grid(2.0, NZ, LZ)
    return SLAdvector(NX, NY, NZ, LX / NX, LY / NY, LX, LY, LZ, z_f, z_c, 2.0, order=6, device="cuda")


def _project(grid, V):
    out = [t.clone() for t in V]
    p = torch.zeros(NX + 2, NY + 2, NZ + 2, dtype=torch.float64, device="cuda")

    def run():
        for o, t in zip(out, V):
            o.copy_(t)
        grid.call("slc_project", *[N.ptr(t) for t in out], N.ptr(p), 0.1, 0.1, N.stream_of(p))

    return run, (*out, p)


def _fields(seed):
    g = torch.Generator().manual_seed(seed)
    shapes = ((NX + 1, NY + 2, NZ + 2), (NX + 2, NY + 1, NZ + 2), (NX + 2, NY + 2, NZ + 1))
    return [torch.randn(s, generator=g, dtype=torch.float64).cuda() for s in shapes]


def test_making_a_handle_launches_nothing():
    before = N.kernel_launches()
    _advector()
    assert N.kernel_launches() == before


def test_first_projection_under_capture():
    V = _fields(1)
    run, want = _project(_advector()._grid, V)
    run()
    captured, got = _project(_advector()._grid, V)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        captured()
    for _ in range(2):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
