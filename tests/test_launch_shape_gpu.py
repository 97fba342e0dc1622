"""The tracking kernel's block size follows the number of particles: results
do not depend on it."""

import numpy as np
import pytest

from sixtracklib_gb300 import lattices

pytestmark = pytest.mark.gpu

# blocks of 32 threads up to nine per SM (43,776 particles), of 64 above
SIZES = [1, 31, 32, 33, 43_776, 43_777, 77_825]


@pytest.mark.parametrize("ring", ["resident", "streamed", "wide"])
def test_results_do_not_depend_on_the_block_size(ring):
    """A lattice resident in shared memory, one streamed through the stages,
    and one whose chunks leave room for fewer blocks (long records)."""
    import torch

    from sixtracklib_gb300.device import DeviceTracker

    lat = {"resident": lattices.fodo_ring, "streamed": lambda: lattices.variant_ring(3, 1200),
           "wide": lambda: lattices.bb_sc_ring(n_bb6d=1, n_bb4d=1, n_sc=2, n_slices=400)}[ring]()
    cols = torch.from_numpy(lattices.gaussian_particles(max(SIZES), seed=9).block.copy()
                            .view(np.int64)).cuda()
    trk = DeviceTracker(lat, "mode=fast")
    for n in SIZES:
        a, b = cols[:, :n].clone(), cols[:, :n].clone()
        assert trk.track_until(a, 2) == 0
        assert DeviceTracker(lat, "mode=fast threads_per_block=128 stages=4").track_until(b, 2) == 0
        assert torch.equal(a, b)
