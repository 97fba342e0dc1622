"""A job's column copies and the upload of tables (csrc/column_copy.h) on the CPU, against a runtime
whose copies to the device land only when their stream is waited for."""

import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "sixtracklib_gb300", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("column_copy") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-I" + CSRC,
                    os.path.join(HERE, "column_copy_check.cpp"), "-o", exe], check=True)

    def run(*args):
        return subprocess.run([exe, *map(str, args)], check=True, capture_output=True,
                              text=True).stdout.strip()

    return run


@pytest.mark.parametrize("direction", ["up", "down"])
@pytest.mark.parametrize("layout", ["single", "packed", "apart", "uneven"])
def test_columns_have_arrived_on_return(check, layout, direction):
    """One copy, pitched copies and column by column; a failing copy is
    reported with none of the others left in flight."""
    assert check(layout, direction, -1) == "ok"
    for fail in (0, 1, 30):
        assert check(layout, direction, fail) == "ok"


def test_tables_have_arrived_on_return(check):
    """Several blocks, an empty one among them."""
    for fail in (-1, 0, 1, 2):
        assert check("blocks", "up", fail) == "ok"
