"""The Gauss restore of links that are not exactly on the group (drifted FP32 links, loaded
ones): the oracle's fields, and no violation left by the oracle's measure, on the host build of
the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc

GAUSS_RMS = 10  # of the observables vector
# the violation of a restored field.  FP64: six terms of order 1, 1e-15 each.  FP32: the
# stored fields' rounding, 3e-8 in six terms, and that of the last sub-steps
RMS = {"f64": 1e-13, "f32": 1e-7}


def state(P, nc, shape, eps, seed=3):
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, seed)
    P.gaussian_efield(shape, E, 0.7, seed + 1)
    return U + eps * np.random.default_rng(5).standard_normal(U.shape), E


def restored(P, H, prec, shape, iterations):
    """Restores H and a copy of its stored state by the oracle; returns both fields and the violation."""
    U, E = H.download()
    H.gauss_restore(1e-14 if prec == "f64" else 0.0, iterations)
    P.gauss_restore(shape, U, E, 1e-14 if prec == "f64" else 0.0, iterations)
    Uh, Eh = H.download()
    return Eh, E, P.observables(shape, Uh, Eh)[GAUSS_RMS]


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("shape", [(4, 5, 6), (3, 2, 2), (4, 3, 5)])  # FP32: pairs, one pair plane, sites
@pytest.mark.parametrize("eps", [0.0, 1e-7, 3e-6, 1e-3])
def test_links_off_the_group(oracle_port, nc, prec, shape, eps):
    P = oracle_port[nc]
    H = hc.HostLattice(nc, prec, shape)
    H.upload(*state(P, nc, shape, eps))
    Eh, E, rms = restored(P, H, prec, shape, 10000 if prec == "f64" else 60)
    assert rms < RMS[prec]
    # FP64: rounding of some hundred sub-steps; FP32: 180 roundings of fields of order 1, whose
    # divergence-free part nothing takes back (6e-8 / 2 * sqrt(180) rms, 5 times that at most)
    assert np.abs(Eh - E).max() < (1e-12 if prec == "f64" else 2e-6)


@pytest.mark.parametrize("nc", [2, 3])
def test_after_fp32_steps(oracle_port, nc):
    """Links as they drift between reunitarisations, restored in FP32 and, copied, in FP64."""
    P, shape = oracle_port[nc], (4, 4, 6)
    H = hc.HostLattice(nc, "f32", shape)
    H.upload(*state(P, nc, shape, 0.0))
    H.leapfrog(0.05, 90)
    H64 = hc.HostLattice(nc, "f64", shape)
    H64.upload(*H.download())
    assert restored(P, H, "f32", shape, 60)[2] < RMS["f32"]
    Eh, E, rms = restored(P, H64, "f64", shape, 10000)
    assert rms < RMS["f64"] and np.abs(Eh - E).max() < 1e-12
