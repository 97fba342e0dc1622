"""The integer- and FP32-pipe parts of the element maps (csrc/intpath.cuh,
csrc/leadkick.cuh, csrc/sckick.cuh) on the GPU,
bit for bit against the oracle (exact policy) and its restatement of the
fast policy, at the edges of the ranges they decide."""

import numpy as np
import pytest

from oracle.pyoracle import Oracle
from sixtracklib_gb300 import lattices
from sixtracklib_gb300.beam_elements import Elements

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracles():
    return {"exact": Oracle(), "fast": Oracle.fast_policy(goertzel=True)}


def _same(lattice, block, oracle, mode):
    import torch

    from sixtracklib_gb300.device import DeviceTracker

    exp = block.copy()
    st = oracle.track_until(lattice.cbuffer.to_image(), exp, 1)
    cols = torch.from_numpy(block.copy().view(np.int64)).cuda()
    assert DeviceTracker(lattice, f"mode={mode}").track_until(cols, 1) == st
    got = cols.cpu().numpy().view(np.uint64)
    nan = np.isnan(exp[:17].view(np.float64)) & np.isnan(got[:17].view(np.float64))
    same = exp == got
    same[:17] |= nan
    assert same.all(), np.argwhere(~same)[:5]


def _momenta():
    """px around every limit of drift_slip: its range 2^-7, zeros, subnormals,
    halves of 2^-52 in t / 2, inf and NaN, and ordinary values."""
    rng = np.random.default_rng(3)
    edge = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0 ** -39, 2.0 ** -26, 2.0 ** -25.5, 2.0 ** -25,
                     np.nextafter(2.0 ** -7, 0), 2.0 ** -7, -(2.0 ** -7), 0.1, 1.5, np.inf, np.nan])
    a, b = np.meshgrid(edge, edge)
    ties = rng.integers(-64, 64, (2, 512)) * 2.0 ** -31
    wide = rng.normal(size=(2, 1024)) * 10.0 ** rng.uniform(-9, -2, (2, 1024))
    return np.concatenate([[a.ravel(), b.ravel()], ties, wide], axis=1)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("p0c", [7e12, 1e9, 3e7])
def test_drift_at_the_edges(oracles, mode, p0c):
    """7 TeV, and momenta at which rvv - u leaves 32 bits (1 GeV) and rvv
    leaves the integer path's range (30 MeV)."""
    px, py = _momenta()
    p = lattices.gaussian_particles(px.size, seed=2, sdelta=3e-3, p0c=p0c)
    p.px[:], p.py[:] = px, py
    p.rpp[:16] = 1.0  # px itself
    e = Elements()
    for length in (1.0, 2.5, 1e-3, 0.0):
        e.Drift(length=length)
    _same(e, p.block, oracles[mode], mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("chi", [1.0, 0.5])
@pytest.mark.parametrize("order", [0, 1, 2, 3, 5])
def test_multipole_zero_coefficients(oracles, mode, chi, order):
    """Zero, minus-zero and nonzero coefficients at every order, coordinates
    that are zeros of both signs, subnormal, huge, inf and NaN: signs of
    zeros included."""
    rng = np.random.default_rng(order)
    v = np.array([0.0, -0.0, 1e-310, 1e-3, -2e-3, 0.7, 1e200, np.inf, np.nan])
    x, y = (a.ravel() for a in np.meshgrid(v, v))
    x, y = np.tile(x, 4), np.tile(y, 4)
    p = lattices.gaussian_particles(x.size, seed=5)
    p.x[:], p.y[:] = x, y
    p.px[:81], p.py[81:162], p.px[162:243] = 0.0, -0.0, -0.0
    p.py[162:243] = 0.0
    p.chi[:] = chi
    for trial in range(8):
        bal = rng.normal(size=2 * order + 2) * 10.0 ** rng.uniform(-3, 0, 2 * order + 2)
        bal[rng.random(bal.size) < 0.5] = 0.0
        if trial < 6:
            bal[1::2] = 0.0  # no skew component
        if trial % 3 == 1:
            bal[bal == 0.0] *= rng.choice([1.0, -1.0], (bal == 0.0).sum())
        e = Elements()
        e.Multipole(order=order, bal=bal)
        _same(e, p.block, oracles[mode], mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("order", [2, 3, 4, 5, 10])
@pytest.mark.parametrize("size", [1e-6, 1e-3, 8e-3, 40e-3])
def test_lead_kick(oracles, mode, order, size):
    """Quadrupoles with multipole errors (lead blocks) of either sign, at
    amplitudes inside, across and beyond their range, on and near the axes;
    one drift between them so that momenta act."""
    rng = np.random.default_rng(order)
    n = 2000
    p = lattices.gaussian_particles(n, seed=order, sx=size, sy=size)
    p.x[:40], p.y[40:80] = 0.0, -0.0
    p.x[80:160] *= 1e-9
    p.y[160:240] *= 10.0 ** rng.uniform(-30, 0, 80)
    p.x[240:260], p.y[240:260] = 0.0, 0.0
    p.px[260:400] = 0.0
    p.chi[1000:1032] = 0.5
    e = Elements()
    for trial in range(24):
        knl = np.zeros(order + 1)
        knl[1] = rng.choice([-1, 1]) * rng.uniform(0.01, 0.05)
        for k in range(2, order + 1):
            knl[k] = rng.normal(0.0, 10.0 ** rng.uniform(-6, -2) * 10.0 ** -k)
        e.Multipole(knl=list(knl))
        e.Drift(length=float(rng.uniform(0.1, 2.0)))
    _same(e, p.block, oracles[mode], mode)


def test_lead_block_follows_the_parameters(oracles):
    """A parameter change that ends or restores the lead of the quadrupole
    term takes effect (the header and the block are made again)."""
    import torch

    from sixtracklib_gb300.autodiff import DifferentiableLattice, apply_values

    e = Elements()
    for k1 in (0.03, -0.02):
        e.Multipole(knl=[0.0, k1, 1e-6, 1e-7], ksl=[0.0, 0.0, 0.0, 0.0])
        e.Drift(length=1.0)
    params = [(0, "knl", 1), (0, "knl", 2), (2, "ksl", 3), (2, "knl", 0)]
    lat = DifferentiableLattice(e, params, "mode=exact")
    p = lattices.gaussian_particles(500, seed=4)
    for values in ([0.03, 1e-6, 0.0, 0.0], [1e-7, 5.0, 0.0, 0.0], [-0.04, -3e-6, 2e-3, 0.0],
                   [0.02, 2e-6, 0.0, 1e-5], [0.015, 1e-6, 0.0, 0.0]):
        lat.set_values(torch.tensor(values, dtype=torch.float64))
        exp = p.block.copy()
        now = apply_values(e, params, values)
        assert oracles["exact"].track_until(now.cbuffer.to_image(), exp, 1) == 0
        cols = torch.from_numpy(p.block.copy().view(np.int64)).cuda()
        assert lat.tracker.track_until(cols, 1) == 0
        assert np.array_equal(cols.cpu().numpy().view(np.uint64), exp)


@pytest.mark.parametrize("sigmas", [(1e-3, 1e-3), (1e-3, 1.2e-3), (1e-3, 0.3e-3)])
@pytest.mark.parametrize("size", [2e-5, 1e-3, 6e-3])
def test_space_charge_kick(oracles, sigmas, size):
    """q-Gaussian kicks 1e-11 of the momenta (pairs) and of the momenta's size
    (FP64), centred and offset: exact mode equal to the oracle, whose libm and
    Faddeeva function differ by 1e-14 of a kick -- 1e-9 of the last bit of a
    momentum where the pairs decide.  The last kick, of a beam 1e9 times as
    intense, is held to 1e-12 of the largest."""
    n = 1500
    p = lattices.gaussian_particles(n, seed=8, sx=size, sy=size)
    p.x[:20], p.y[20:40] = 0.0, 0.0
    p.px[40:60], p.py[60:80] = 0.0, 1e-15
    p.px[80:100] = 1e-18
    e = Elements()
    for k, (x_co, y_co) in enumerate([(0.0, 0.0), (1e-5, 0.0), (0.0, -2e-5), (0.0, 0.0)]):
        e.SCQGaussProfile(number_of_particles=1e11 * (1 + k), bunchlength_rms=0.1,
                          sigma_x=sigmas[0], sigma_y=sigmas[1], length=0.1, x_co=x_co, y_co=y_co,
                          min_sigma_diff=1e-10, q_param=1.0, enabled=1)
    small = p.block.copy().view(np.float64)
    lost = slice(0, 100)  # momenta at or below the kick's size: no last bit to compare
    import torch

    from sixtracklib_gb300.device import DeviceTracker

    exp = p.block.copy()
    oracles["exact"].track_until(e.cbuffer.to_image(), exp, 1)
    for mode in ("exact", "fast"):
        cols = torch.from_numpy(p.block.copy().view(np.int64)).cuda()
        assert DeviceTracker(e, f"mode={mode}").track_until(cols, 1) == 0
        got = cols.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[:, 100:], exp[:, 100:])
        kick = got[8:10, lost].view(np.float64) - small[8:10, lost]
        ref = exp[8:10, lost].view(np.float64) - small[8:10, lost]
        assert np.abs(kick - ref).max() <= 1e-12 * np.abs(ref).max()
    strong = Elements()
    strong.SCQGaussProfile(number_of_particles=1e20, bunchlength_rms=0.1, sigma_x=sigmas[0],
                           sigma_y=sigmas[1], length=0.1, min_sigma_diff=1e-10, q_param=1.0,
                           enabled=1)
    exp = p.block.copy()
    oracles["exact"].track_until(strong.cbuffer.to_image(), exp, 1)
    cols = torch.from_numpy(p.block.copy().view(np.int64)).cuda()
    assert DeviceTracker(strong, "mode=exact").track_until(cols, 1) == 0
    got = cols.cpu().numpy().view(np.uint64)
    ref = exp[8:10].view(np.float64) - small[8:10]
    assert np.abs(got[8:10].view(np.float64) - exp[8:10].view(np.float64)).max() <= \
        1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("mode", ["exact", "fast"])
def test_products_on_the_integer_pipes(oracles, mode):
    """More particles than two warps per scheduler (40,000): the products of
    drifts and leading quadrupoles run on the integer pipes."""
    px, py = _momenta()
    n = 40_000
    p = lattices.gaussian_particles(n, seed=6, sdelta=3e-3)
    p.px[:] = np.resize(px, n)
    p.py[:] = np.resize(py, n)
    p.x[::7], p.y[::11] = 0.0, -0.0
    e = Elements()
    for k in range(6):
        e.Drift(length=1.0 + k)
        e.Multipole(knl=[0.0, 0.03 - 0.01 * k])
        e.Multipole(knl=[0.0, 0.01 + 0.01 * k, 1e-6, 1e-7, -1e-8])
    _same(e, p.block, oracles[mode], mode)
