"""The walk over short lattices: drifts and multipoles at the start, at the
end and next to other elements, particles lost in each of them, whole turns
and sections, against the oracle bit for bit."""

import numpy as np
import pytest

from sixtracklib_gb300 import lattices
from sixtracklib_gb300.beam_elements import Elements

pytestmark = pytest.mark.gpu


def lattice(order):
    e = Elements()
    rng = np.random.default_rng(len(order))
    for o in order:
        if o == "d":
            e.Drift(length=1.5)
        elif o == "c":
            e.Cavity(voltage=3e6, frequency=4e8, lag=170.0)
        elif o == "b":
            e.LimitRect(min_x=-0.015, max_x=0.015, min_y=-0.02, max_y=0.02)
        elif o == "k":  # a kick that sends particles past the limit of every drift
            e.Multipole(knl=[0.3, 0.0], ksl=[0.0, 0.0])
        elif o == "l":  # a quadrupole with small errors
            e.Multipole(knl=[0.0, 0.02, *rng.normal(0, 1e-4, 6)], ksl=[0.0] + [1e-6] * 7)
        else:
            e.Multipole(knl=[0.0, 0.02])
    return e


# 257: latency-bound walk; 40,001: above two warps per scheduler
@pytest.mark.parametrize("n", [257, 40_001])
@pytest.mark.parametrize("order", ["d", "q", "l", "b", "dq", "qd", "bq", "lb", "db", "cd", "lc",
                                   "kdd", "kdbd", "dkddddb", "cqldbdlqc", "dldqblkddc"])
def test_short_lattices_like_the_oracle(oracle, order, n):
    import torch

    from sixtracklib_gb300.device import DeviceTracker

    e = lattice(order)
    img = e.cbuffer.to_image()
    blk = lattices.gaussian_particles(n, seed=3).block.copy()
    blk.view(np.float64)[6, : n // 4] = np.linspace(-1.2, 1.2, n // 4)
    trk = DeviceTracker(e, "mode=exact")
    for line in (None, (len(order) // 2, len(order))):
        exp = blk.copy()
        cols = torch.from_numpy(blk.copy().view(np.int64)).cuda()
        if line is None:
            want, got = oracle.track_until(img, exp, 3), trk.track_until(cols, 3)
        else:
            want, got = oracle.track_line(img, exp, *line), trk.track_line(cols, *line, False)
        assert got == want
        out = cols.cpu().numpy().view(np.uint64)
        np.testing.assert_array_equal(out, exp)
    if "k" in order:
        assert (exp[20] == 0).any()
