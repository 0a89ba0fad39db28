"""The paired step of small lattices (three threads a pair) against the one-thread kernel."""
import numpy as np
import pytest

import topologicalcymsolver_gb300 as tcym

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [2, 3])
# fewer pairs than a block, a ragged last block, the largest that splits and the first that does not
@pytest.mark.parametrize("shape", [(2, 3, 2), (5, 7, 6), (33, 5, 10), (50, 50, 20), (51, 50, 20), (61, 30, 36)])
def test_split_and_whole_steps_same_bits(ctx, nc, shape):
    """A tiling fixed by the caller takes the one-thread kernel at every size: the same bits as the
    library's choice for leapfrog, Langevin and flow."""
    out = []
    for tile in (None, (8, 16)):
        lat = tcym.Lattice(ctx, nc, shape, tcym.FP32)
        lat.set_tile(*(tile or (0, 0)))
        lat.random_links(0.5, 3)
        lat.gaussian_efield(0.7, 4)
        lat.leapfrog(0.05, 3)
        lat.langevin(0.02, 1.0, 0.6, 7, 5, 2)
        lat.flow(0.02, 2)
        out.append(lat.download())
        lat.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
