"""Checkerboard flow of lattices longer than a launch has tiles along y and z."""
import numpy as np
import pytest

import topologicalcymsolver_gb300 as tcym

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 524296), (2, 262152, 4), (2, 4, 524280)])  # beyond in z, in y, the last within
def test_checkerboard(ctx, oracle_port, shape):
    """One sweep: FP32 links' rounding, 6 updates of entries below 1."""
    V = int(np.prod(shape))
    U = np.zeros((V, 3, 4))
    oracle_port[2].random_links(shape, U, 0.5, 9)
    lat = tcym.Lattice(ctx, 2, shape, tcym.FP32)
    lat.upload(U)
    lat.flow(0.05, 1, tcym.FLOW_CHECKERBOARD)
    oracle_port[2].flow_checkerboard(shape, U, 0.05, 1)
    assert np.abs(lat.download()[0] - U).max() < 2e-6
    lat.close()
