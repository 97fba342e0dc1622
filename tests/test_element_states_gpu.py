"""Element-by-element tracking of particles whose state is neither 0 nor 1:
an aperture keeps the lowest bit of a state, any other map leaves it, and a
particle goes on while its state is 1 -- as in the oracle."""

import numpy as np
import pytest

from oracle.pyoracle import EbeConfig, Oracle
from sixtracklib_gb300 import (ParticlesSet, TriCub_buffer_create_assign_address_item,
                               lattices)
from sixtracklib_gb300.beam_elements import Elements
from sixtracklib_gb300.trackjob import TrackJob

from .tricub_cases import _grid

pytestmark = pytest.mark.gpu

GRID = (8, 8, 5, 2e-3, 2e-3, 0.1, -7e-3, -7e-3, -0.2)
STATES = [1, 0, 2, 3, 5, 6, -1, -2]


def lattice(kind, data=None):
    e = Elements()
    if kind == "drift":
        e.Drift(length=1.0)
    elif kind == "exact drift":
        e.DriftExact(length=1.0)
    elif kind == "rect":
        e.LimitRect(min_x=-1e-3, max_x=1e-3, min_y=-1e-3, max_y=1e-3)
    elif kind == "ellipse":
        e.LimitEllipse(a_squ=1e-6, b_squ=1e-6)
    elif kind == "rect ellipse":
        e.LimitRectEllipse(max_x=1e-3, max_y=1e-3, a_squ=1e-6, b_squ=1e-6)
    elif kind == "multipole":
        e.Multipole(knl=[0.0, 0.02])
    else:
        e.TriCub(data=data, length=1.0)
    e.Drift(length=0.5)
    if kind == "tricub and beams":  # the kernel with every map
        e.SCCoasting(number_of_particles=0.0, circumference=1000.0, sigma_x=1e-3, sigma_y=1.5e-3,
                     length=1.0)
    else:
        e.Multipole(knl=[0.0, 0.01])
    if kind.startswith("tricub"):
        _grid(e, np.random.default_rng(1), *GRID)
    return e


@pytest.mark.parametrize("kind", ["drift", "exact drift", "rect", "ellipse", "rect ellipse",
                                  "multipole", "tricub", "tricub and beams"])
def test_states_like_the_oracle(kind):
    e = lattice(kind)
    n = 40 * len(STATES)
    q = lattices.gaussian_particles(n, seed=3, sx=1e-3, sy=1e-3, sz=0.03)
    q.state[:] = np.tile(STATES, 40)
    ps = ParticlesSet()
    p = ps.Particles(num_particles=n)
    p.set_block(q.block)
    job = TrackJob(e, ps, until_turn_elem_by_elem=2,
                   config_str="mode=exact track_tricub=enabled")
    if kind.startswith("tricub"):  # the job's TriCub data come from a stored buffer
        tables = Elements()
        _grid(tables, np.random.default_rng(1), *GRID)
        bid = job.add_stored_buffer(cbuffer=tables)
        assert TriCub_buffer_create_assign_address_item(job, 0, bid, 0)
        job.commit_address_assignments()
        job.assign_all_addresses()
    got_status = job._lib.st_TrackJob_track_elem_by_elem(job.ptr_st_track_job, 2)
    job.collect()
    got = job.output.cbuffer.get_object(0).block
    ne = len(e)
    exp, exp_out = q.block.copy(), np.zeros_like(got)
    oracle = Oracle()
    oracle.set_track_flags(tricub=2)
    try:
        want_status = oracle.track_elem_by_elem(
            lattice(kind, data=3).cbuffer.to_image(), exp,
            EbeConfig(0, n, ne, 2, 0, 0, 0, n - 1, ne - 1, 1, 1), exp_out, 2)
    finally:
        oracle.set_track_flags()
    assert got_status == want_status
    np.testing.assert_array_equal(p.block, exp)
    np.testing.assert_array_equal(got, exp_out)
