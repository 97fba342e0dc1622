"""The kicks evaluated in pairs of floats (csrc/leadkick.cuh,
csrc/sckick.cuh) on the GPU, bit for bit against the oracle at the ends of the range that they
accept."""

import numpy as np
import pytest

from oracle.pyoracle import Oracle
from sixtracklib_gb300 import lattices
from sixtracklib_gb300.beam_elements import Elements

pytestmark = pytest.mark.gpu


def _same(lattice, block, oracle, mode):
    import torch

    from sixtracklib_gb300.device import DeviceTracker

    exp = block.copy()
    oracle.track_until(lattice.cbuffer.to_image(), exp, 1)
    cols = torch.from_numpy(block.copy().view(np.int64)).cuda()
    assert DeviceTracker(lattice, f"mode={mode}").track_until(cols, 1) == 0
    got = cols.cpu().numpy().view(np.uint64)
    assert np.array_equal(got, exp), np.argwhere(got != exp)[:5]


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_lead_kick_at_small_coordinates(mode):
    """One plane's coordinates and momenta from 1e-40 m up and zero, the other's
    of a beam; blocks of 32 particles of one size, so that warps are all in
    range or not."""
    rng = np.random.default_rng(23)
    n = 32 * 64
    p = lattices.gaussian_particles(n, seed=23)
    size = np.repeat(10.0 ** -np.linspace(3.0, 40.0, 32), 32)
    size[:32] = 0.0
    for k, (q, pq) in enumerate(((p.y, p.py), (p.x, p.px))):
        part = slice(k * n // 2, (k + 1) * n // 2)
        q[part] = size * rng.choice([-1.0, 1.0], n // 2)
        pq[part] = 0.01 * size * rng.normal(size=n // 2)
    e = Elements()
    for trial in range(12):
        knl = np.zeros(2 + trial % 6 + 1)
        knl[1] = rng.choice([-1, 1]) * rng.uniform(0.01, 0.05)
        for k in range(2, knl.size):
            knl[k] = rng.normal(0.0, 10.0 ** rng.uniform(-4, -1))
        e.Multipole(knl=list(knl))
    _same(e, p.block, Oracle() if mode == "exact" else Oracle.fast_policy(goertzel=True), mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("sigma", [1e-5, 2e-5, 5e-5, 1e-4])
def test_round_space_charge_near_the_axis(mode, sigma):
    """Particles on both sides of 1e-10 m from the axis, where the field changes
    its form, with momenta whose last bit is of the kick's size (1e-14 of a
    kick, by which the oracle's libm differs, is far below it)."""
    rng = np.random.default_rng(29)
    n = 32 * 64
    p = lattices.gaussian_particles(n, seed=29)
    r = np.repeat(10.0 ** np.linspace(-12.0, -9.0, 64), 32)
    for q in (p.x, p.y, p.px, p.py):
        q[:] = rng.choice([-1.0, 1.0], n)
    p.x[:] *= r * rng.uniform(0.5, 1.0, n)
    p.y[:] *= r * rng.uniform(0.5, 1.0, n)
    p.px[:] *= 10.0 ** rng.uniform(-7, -1, n)
    p.py[:] *= 10.0 ** rng.uniform(-7, -1, n)
    e = Elements()
    for k in range(3):
        e.SCQGaussProfile(number_of_particles=1e11 * (1 + k), bunchlength_rms=0.1, sigma_x=sigma,
                          sigma_y=sigma, length=0.1, min_sigma_diff=1e-10, q_param=1.0, enabled=1)
    _same(e, p.block, Oracle(), mode)
