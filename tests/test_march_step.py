"""The FP64 step in blocks that share their plaquettes (tcym_march.cuh): every tiling
gives the same bits, and the oracle's step, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc

# tilings (tx, ty, planes a block, threads): one site, ragged, as wide as the lattice, larger
# than it, one plane and every plane a block, fewer threads than tasks, the rule's own choices
TILINGS = [(1, 1, 1, 32), (3, 2, 2, 32), (5, 3, 3, 96), (8, 8, 64, 224), (2, 7, 1, 64), (0, 0, 0, 152), (0, 0, 0, 0),
           (0, 0, 0, 4)]
# FP64: rounding of a step, 1e-14 of the fields; FP32 storage: one rounding of U and E, 1e-6
TOL = {"f64": 1e-13, "f32": 1e-6}


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 4, 3), (9, 5, 7), (17, 3, 2)])
def test_tilings_same_bits_and_oracle(oracle_port, nc, prec, shape):
    P = oracle_port[nc]
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, 3)
    P.gaussian_efield(shape, E, 0.7, 4)
    out = []
    for t in TILINGS:
        H = hc.HostLattice(nc, prec, shape)
        H.upload(U, E)
        H.march(0.05, *t)
        out.append(H.download())
    for Uh, Eh in out[1:]:
        assert np.array_equal(Uh, out[0][0]) and np.array_equal(Eh, out[0][1])
    P.leapfrog(shape, U, E, 0.05, 1)
    assert np.abs(out[0][0] - U).max() < TOL[prec]
    assert np.abs(out[0][1] - E).max() < TOL[prec] * np.abs(E).max()
