"""The integer-pipe parts of the element maps (csrc/intpath.cuh) on the GPU,
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
