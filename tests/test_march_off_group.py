"""The FP64 step of links that are not exactly on the group (copied from FP32, loaded with few
digits), in blocks that share their plaquettes, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc

# tilings as in test_march_step: ragged, every plane a block, the rule's own choices
TILINGS = [(3, 2, 2, 32), (8, 8, 64, 224), (0, 0, 0, 152), (0, 0, 0, 0)]


def step(P, nc, shape, spoil, tilings):
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, 3)
    P.gaussian_efield(shape, E, 0.7, 4)
    spoil(U)
    out = []
    for t in tilings:
        H = hc.HostLattice(nc, "f64", shape)
        H.upload(U, E)
        H.march(0.05, *t)
        out.append(H.download())
    for Uh, Eh in out[1:]:
        assert np.array_equal(Uh, out[0][0]) and np.array_equal(Eh, out[0][1])
    P.leapfrog(shape, U, E, 0.05, 1)
    return out[0][0] - U, out[0][1] - E


def noise(eps):
    def spoil(U):
        U += eps * np.random.default_rng(5).standard_normal(U.shape)
    return spoil


@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 5, 7), (17, 3, 2)])
@pytest.mark.parametrize("eps", [0.0, 1e-12, 1e-7, 3e-6, 3e-5, 1e-3, 0.3])  # both sides of the series' limit
def test_su2_is_exact_for_any_quaternion(oracle_port, shape, eps):
    """Rounding of a step: 1e-14 of links and fields of order 1."""
    dU, dE = step(oracle_port[2], 2, shape, noise(eps), TILINGS)
    assert np.abs(dU).max() < 1e-14 and np.abs(dE).max() < 1e-14


def test_su2_zero_links(oracle_port):
    """A zero link's loops are zero, not NaN."""
    def spoil(U):
        U[7, 1], U[20, 2], U[33, 0] = 0.0, 0.0, 0.0
    dU, dE = step(oracle_port[2], 2, (4, 3, 5), spoil, TILINGS)
    assert np.abs(dU).max() < 1e-14 and np.abs(dE).max() < 1e-14


@pytest.mark.parametrize("shape", [(9, 5, 7), (6, 5, 8)])
@pytest.mark.parametrize("eps", [1e-12, 1e-7, 3e-6, 1e-3])
def test_su3_no_further_off_than_staples(oracle_port, shape, eps):
    """SU(3): V^dagger for V^-1 is off by eps.  A step of one site a thread by staples of group
    elements (third rows from the first two) is 0.244 eps off in E (dt 0.05, rms)."""
    _, dE = step(oracle_port[3], 3, shape, noise(eps), TILINGS)
    assert np.sqrt((dE ** 2).mean()) < 0.244 * eps
