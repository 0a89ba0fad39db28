"""The FP32 measurements in site pairs of links that are not exactly on the group, on the host
build of the device code: the per-site code (odd nz takes it) and the oracle on the stored state."""
import numpy as np
import pytest

from tests import _hostcheck as hc


def lattice(P, nc, shape, eps, prec="f32"):
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, 3)
    P.gaussian_efield(shape, E, 0.7, 4)
    H = hc.HostLattice(nc, prec, shape)
    H.upload(U + eps * np.random.default_rng(5).standard_normal(U.shape), E)
    return H


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 4), (4, 4, 6)])
@pytest.mark.parametrize("eps", [0.0, 3e-6, 1e-3, 0.1])
def test_sample(oracle_port, nc, shape, eps):
    """E^2, B^2 and E.B: at most 96 sites' FP32 terms of order 1 to 10, 1e-6 each at most, of
    either sign."""
    H = lattice(oracle_port[nc], nc, shape, eps)
    o, r = H.edotb_pair(), oracle_port[nc].observables(shape, *H.download())
    for k in [*range(9), 13]:
        assert abs(o[k] - r[k]) <= 1e-5 * max(1.0, abs(r[k])), k


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("restore", [False, True])
@pytest.mark.parametrize("eps", [0.0, 3e-6, 1e-3])
def test_gauss_violation(oracle_port, nc, restore, eps):
    """The pairs' sums of six FP32 terms, exact but for the last rounding (6e-8 of the violation,
    which a restore cancels to 1e-7), as the per-site sums in FP64."""
    H = lattice(oracle_port[nc], nc, (4, 4, 6), eps)
    if restore:
        H.gauss_restore(0.0, 60)
    a, b = H.gauss(True), H.gauss(False)
    assert (np.abs(a - b) <= 1e-7 * np.abs(b) + 1e-14).all()


@pytest.mark.parametrize("nc", [2, 3])
def test_plaquette_term_as_exact_as_per_site(oracle_port, nc):
    """B^2 of pairs against the oracle on the stored state, over 40 lattices: no further off (rms) than the per-site
    code, whose last product is rounded near 1."""
    P, shape, off = oracle_port[nc], (8, 8, 8), []
    for seed in range(40):
        U, E = np.zeros((512, 3, hc.NM[nc])), np.zeros((512, 3, hc.NA[nc]))
        P.random_links(shape, U, 0.3, seed)
        H = hc.HostLattice(nc, "f32", shape)
        H.upload(U, E)
        r = P.observables(shape, *H.download())[6:9]
        off.append([H.edotb_pair()[6:9] / r - 1, H.observables(8)[6:9] / r - 1])
    pairs, sites = np.sqrt((np.array(off) ** 2).mean((0, 2)))
    assert pairs <= sites
