"""Checkerboard flow of FP32 lattices: pairs of one parity (nz / 2 even) and the per-site
sub-sweeps (nz / 2 odd) against the oracle, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc


@pytest.mark.parametrize("nc", [2, 3])
# two pair planes (both at the seam), more, one (nz 2), odd halves
@pytest.mark.parametrize("shape", [(4, 4, 4), (2, 6, 8), (6, 4, 12), (4, 4, 2), (4, 2, 6)])
def test_checkerboard_against_oracle(oracle_port, nc, shape):
    """Four sweeps: 24 updates of FP32 links, each rounded to 6e-8 of entries below 1."""
    P = oracle_port[nc]
    V = int(np.prod(shape))
    U = np.zeros((V, 3, hc.NM[nc]))
    P.random_links(shape, U, 0.5, 9)
    H = hc.HostLattice(nc, "f32", shape)
    H.upload(U, None)
    H.flow_checkerboard(0.05, 4)
    P.flow_checkerboard(shape, U, 0.05, 4)
    assert np.abs(H.download()[0] - U).max() < 2e-6
