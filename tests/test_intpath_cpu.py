"""The integer- and FP32-pipe parts of the element maps (csrc/intpath.cuh,
csrc/leadkick.cuh, csrc/sckick.cuh), on the CPU: every value they decide has the bits of the
FP64 sequence they stand for."""

import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sixtracklib_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("intpath") / "check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", "-I" + CSRC,
                    os.path.join(HERE, "intpath_check.cpp"), "-o", exe], check=True)

    def run(what, n, seed):
        out = subprocess.run([exe, what, str(n), str(seed)], check=True, capture_output=True,
                             text=True).stdout
        return [int(v) for v in out.split()]

    return run


@pytest.mark.parametrize("what", ["ordinary", "wide", "ties", "special"])
def test_drift_slip_has_the_fp64_bits(check, what):
    """Both policies' rvv - (1 + (xp^2 + yp^2) / 2)."""
    n, undecided, different = check(what, 2_000_000, 7)
    print(f"{what}: {undecided} of {n} left to the FP64 sequence")
    assert different == 0
    assert undecided < n


@pytest.mark.parametrize("what", ["lead exact", "lead fast", "lead exact wide", "lead fast wide"])
def test_lead_kick_has_the_fp64_bits(check, what):
    """Both policies' kicks of quadrupoles with multipole errors, at 1 mm with
    small errors and at 5 mm with errors 100 times larger."""
    n, undecided, different = check(what, 400_000, 11)
    print(f"{what}: {undecided} of {n} left to the FP64 sequence")
    assert different == 0
    assert undecided < n


@pytest.mark.parametrize("beam", ["round", "tall", "flat"])
@pytest.mark.parametrize("where", ["sigma", "wide", "core"])
def test_space_charge_kick_within_its_bounds(check, beam, where):
    """The pair evaluation's bounds hold the kick (the CERN algorithm's
    Faddeeva function in long double), at 1, 5 and 0.02 sigma rms."""
    n, undecided, different = check(f"sc {beam} {where}", 50_000, 5)
    print(f"{beam} {where}: {undecided} of {n} left to the FP64 evaluation")
    assert different == 0
    assert undecided < n


@pytest.mark.parametrize("operands", ["ordinary", "bits", "short", "special"])
def test_product_is_the_rounded_one(check, operands):
    """mul_rn: significands of any length, halves, zeros of both signs,
    subnormals, infinities and NaN (those it refuses)."""
    n, undecided, different = check(f"product {operands}", 2_000_000, 3)
    print(f"{operands}: {undecided} of {n} left to the FP64 product")
    assert different == 0
    assert undecided < n
