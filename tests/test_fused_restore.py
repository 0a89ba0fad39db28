"""The fused Gauss restore (a sub-step's update and the next deviation in one pass) against
the oracle, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("prec", ["f64", "f32"])
# pairs: one plane (nz 2), two; odd nz (FP32: the two-kernel restore); extents of 2 and 3
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 4), (4, 5, 6), (4, 3, 5)])
@pytest.mark.parametrize("iterations", [0, 1, 2, 5])
def test_mid_restore_fields(oracle_port, nc, prec, shape, iterations):
    """After a fixed number of iterations, odd ones ending in the spare buffer: FP64 to a few
    rounding errors a sub-step (15 of them, 1e-13), FP32 likewise (2e-6 of E of order 1)."""
    P = oracle_port[nc]
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, 3)
    P.gaussian_efield(shape, E, 0.7, 4)
    H = hc.HostLattice(nc, prec, shape)
    H.upload(U, E)
    assert H.gauss_restore(0.0, iterations) == iterations
    P.gauss_restore(shape, U, E, 0.0, iterations)
    Uh, Eh = H.download()
    assert np.abs(Eh - E).max() < (1e-13 if prec == "f64" else 2e-6)
