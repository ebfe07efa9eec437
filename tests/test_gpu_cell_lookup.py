"""The cell lookup of the wall-normal stencils (half_cell: bins over the height
and one comparison; at gamma 6 the lowest half cell would need too many bins
and the kernels invert the map) against the oracle's inversion of the tanh map:
linear interpolation of the node index, at random heights and on and beside
every face and centre of the lower half, where a height is known to far less
than a cell.

Linear weights lie in [0, 1], so rounding stays within some units of 1e-16 of
the largest index, and beside an edge the two cells' interpolants differ by the
height's own rounding over the cell: 1e-12 of the largest index leaves both a
wide margin."""

import numpy as np
import pytest
import torch

from oracle.slbdf2 import OracleAdvector, generate_grid
from slchannel_b200.semilag import SLAdvector

pytestmark = pytest.mark.gpu

NX, NY, LX, LY, LZ = 10, 8, 2.0, 1.5, 2.0


@pytest.mark.parametrize("gamma", [0.5, 2.0, 6.0])
@pytest.mark.parametrize("stretching", ["symmetric", "bottom"])
@pytest.mark.parametrize("nz", [6, 33, 130])
def test_lookup_matches_the_inverted_map(gamma, stretching, nz):
    zf, zc, _, _ = generate_grid(gamma, nz, LZ, stretching)
    args = (NX, NY, nz, LX / NX, LY / NY, LX, LY, LZ)
    orc = OracleAdvector(*args, zf, zc, gamma, stretching_type=stretching, order=4)
    adv = SLAdvector(*args, torch.from_numpy(zf), torch.from_numpy(zc), gamma, stretching_type=stretching,
                     order=4, device="cuda")
    rng = np.random.default_rng(nz)
    edges = np.concatenate([zf, zc[1:-1]])
    edges = edges[edges < 0.5 * LZ]
    z = np.concatenate([rng.uniform(0.0, 0.5 * LZ, 400), edges, np.nextafter(edges, -1.0), np.nextafter(edges, 9.0)])
    x, y = rng.uniform(0.0, LX, z.size), rng.uniform(0.0, LY, z.size)
    t = [torch.from_numpy(a).cuda() for a in (x, y, z)]
    for comp in "uvw":
        spec = adv.spec[comp]
        buf = np.broadcast_to(np.arange(spec.NZ, dtype=np.float64), (NX, NY, spec.NZ)).copy()
        got = adv._apply_iw(torch.from_numpy(buf).cuda(), adv._build_iw(spec, *t, 2, count_clamp=True))
        want, _ = orc.interp(comp, 2, buf, x, y, z, count_clamp=True)
        err = float(np.abs(got.cpu().numpy() - want).max())
        assert err <= 1e-12 * spec.NZ, (comp, err)
