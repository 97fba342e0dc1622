"""The kicks evaluated in pairs of floats (csrc/leadkick.cuh,
csrc/sckick.cuh), on the CPU, over the whole range of coordinates and momenta
that they accept: what they decide has the FP64 sequence's bits."""

import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sixtracklib_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("kick_bounds") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", "-I" + CSRC,
                    os.path.join(HERE, "kick_bounds_check.cpp"), "-o", exe], check=True)

    def run(what, n, seed):
        out = subprocess.run([exe, what, str(n), str(seed)], check=True, capture_output=True,
                             text=True).stdout
        return [int(v) for v in out.split()]

    return run


@pytest.mark.parametrize("what", ["lead exact", "lead fast"])
def test_lead_kick_at_small_coordinates(check, what):
    """One coordinate down to 1e-40 m, momenta of the kick's own size: there the
    last bits of the corrections to u_1 x and u_1 y show."""
    n, undecided, different = check(what, 1_000_000, 17)
    print(f"{what}: {undecided} of {n} left to the FP64 sequence")
    assert different == 0
    assert undecided < n


def test_round_space_charge_near_the_axis(check):
    """Beams of 1 um to 1 mm, particles from 1e-13 to 1e-8 m: the field has
    another form within 1e-10 m of the axis."""
    n, undecided, different = check("near axis", 1_000_000, 19)
    print(f"{undecided} of {n} left to the FP64 evaluation")
    assert different == 0
    assert undecided < n


@pytest.mark.parametrize("beam", ["round", "elliptic"])
def test_space_charge_bounds_over_the_bunch(check, beam):
    """The longitudinal exponent over its whole range, beams of 10 nm to 1 cm
    and bunches of 1 mm to 0.3 m: the bounds hold every kick."""
    n, undecided, different = check(f"tails {beam}", 500_000, 31)
    print(f"{beam}: {undecided} of {n} left to the FP64 evaluation")
    assert different == 0
    assert undecided < n


def test_exponential_table(check):
    """Its entries, and their alignment for a load of 8 bytes."""
    assert check("table", 32, 0) == [32, 0, 0]
