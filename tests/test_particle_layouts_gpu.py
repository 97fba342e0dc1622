"""Particle sets whose columns follow one another, lie at one distance or in
no order: pushed, tracked, collected and recorded alike."""

import numpy as np
import pytest

from sixtracklib_gb300 import lattices
from sixtracklib_gb300.cbuffer import CObject
from sixtracklib_gb300.particles import NUM_COLUMNS, TYPE_PARTICLE, Particles, ParticlesSet

LAYOUTS = ["packed", "spaced", "reversed", "shuffled"]


def laid_out(block, how):
    n = block.shape[1]
    pitch = n + 5 if how == "spaced" else n
    order = {"reversed": np.arange(NUM_COLUMNS)[::-1],
             "shuffled": np.random.default_rng(1).permutation(NUM_COLUMNS)}.get(
                 how, np.arange(NUM_COLUMNS))
    words = np.zeros(22 + NUM_COLUMNS * pitch, dtype=np.uint64)
    words[0] = n
    words[1:22] = 22 + order * pitch
    for c in range(NUM_COLUMNS):
        words[22 + order[c] * pitch: 22 + order[c] * pitch + n] = block[c]
    return CObject(TYPE_PARTICLE, words, list(range(1, 22)))


def columns(p):
    return np.stack([p.column(c).view(np.uint64) for c in range(NUM_COLUMNS)])


@pytest.mark.parametrize("how", LAYOUTS)
@pytest.mark.parametrize("n", [1, 3, 257])
def test_block_and_set_block(how, n):
    rng = np.random.default_rng(n)
    block = rng.integers(1, 2**60, (NUM_COLUMNS, n)).astype(np.uint64)
    other = rng.integers(1, 2**60, (NUM_COLUMNS, n)).astype(np.uint64)
    p = Particles._from_cobject(laid_out(block, how))
    assert np.array_equal(p.block, block)
    p.set_block(other)
    assert np.array_equal(columns(p), other)
    if n == 3:
        with pytest.raises(ValueError):
            p.set_block(other[:, :2])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 1000])
@pytest.mark.parametrize("sets", [(h,) for h in LAYOUTS] + [tuple(LAYOUTS)])
def test_jobs_do_not_depend_on_the_layout(sets, n):
    from sixtracklib_gb300.device import DeviceTracker
    from sixtracklib_gb300.trackjob import TrackJob
    import torch

    lat = lattices.fodo_ring()
    blocks = [lattices.gaussian_particles(n + 2 * k, seed=5 + k).block.copy()
              for k in range(len(sets))]
    ps = ParticlesSet()
    for b, how in zip(blocks, sets):
        ps.cbuffer.add_raw(laid_out(b, how))
    job = TrackJob(lat, ps, particle_set_indices=range(len(sets)))
    for turns in (1, 2):
        for k, b in enumerate(blocks):  # pushed again: the job's copy is overwritten
            ps.cbuffer.get_object(k).set_block(b)
        job.push_particles()
        assert job.track_until(turns) == 0
        job.collect_particles()
        for k, b in enumerate(blocks):
            cols = torch.from_numpy(b.copy().view(np.int64)).cuda()
            assert DeviceTracker(lat).track_until(cols, turns) == 0
            assert np.array_equal(columns(ps.cbuffer.get_object(k)),
                                  cols.cpu().numpy().view(np.uint64))
