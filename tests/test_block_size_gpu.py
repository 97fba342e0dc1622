"""The block size that a CUDA job reports is the one its tracking kernel runs
with: 32 threads while nine such blocks per SM hold the particles, 64 above,
or what the configuration says."""

import pytest

from sixtracklib_gb300 import ParticlesSet, lattices
from sixtracklib_gb300.trackjob import CudaTrackJob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, config, threads", [
    (1, "", 32), (1_000, "", 32), (43_776, "", 32), (43_777, "", 64), (60_000, "", 64),
    (1_000, "cuda.threads_per_block = 96", 96),
    (1_000, "cuda.threads_per_block = 96\ncuda.track_threads_per_block = 160", 160)])
def test_reported_block_size(n, config, threads):
    ps = ParticlesSet()
    p = ps.Particles(num_particles=n)
    p.set_block(lattices.gaussian_particles(n, seed=1).block)
    job = CudaTrackJob(lattices.variant_ring(3, 1200), ps, config_str=config)
    assert job.default_track_threads_per_block == threads
    assert job.track_until(1) == 0
