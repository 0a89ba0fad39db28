"""The FP32 formats' reunitarisation (increments as sums of a value and its error) against
the FP64 projection rounded once, bit for bit, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc

# deviations of the stored rows: rounding, a long run, the edge of the increment form, beyond it
DRIFTS = [0.0, 3e-6, 1.5e-5, 2e-4, 4e-3]


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [(16, 16, 12), (3, 3, 3), (8, 5, 2)])  # odd volume: a padded pair
@pytest.mark.parametrize("drift", DRIFTS)
def test_projection_is_the_fp64_one_rounded_once(oracle_port, nc, shape, drift):
    """Each entry is the FP64 projection's, rounded once: equal to the last bit."""
    P = oracle_port[nc]
    V = int(np.prod(shape))
    U = np.zeros((V, 3, hc.NM[nc]))
    P.random_links(shape, U, 0.9, 5)
    U *= 1 + drift * np.random.default_rng(3).uniform(-1, 1, size=U.shape)
    A, B = hc.HostLattice(nc, "f32", shape), hc.HostLattice(nc, "f32", shape)
    for H in (A, B):
        H.upload(U, None)
    A.reunitarize()
    B.reunitarize_fp64()
    # an odd volume's pad lane holds no site: compare the sites
    assert np.array_equal(A.download()[0], B.download()[0])


@pytest.mark.parametrize("nc", [2, 3])
def test_projection_of_a_broken_link_is_the_fp64_one(oracle_port, nc):
    """NaN and infinite entries, and a zero link, take the FP64 projection lane by lane:
    the partner site of the pair and every other link are as without them."""
    shape, P = (4, 4, 4), oracle_port[nc]
    U = np.zeros((64, 3, hc.NM[nc]))
    P.random_links(shape, U, 0.9, 6)
    bad = U.copy()
    bad[3, 1, 0], bad[10, 0, 0], bad[40, 2, :] = np.nan, np.inf, 0.0
    out = []
    for V in (U, bad):
        H = hc.HostLattice(nc, "f32", shape)
        H.upload(V, None)
        H.reunitarize()
        out.append(H.download()[0])
    keep = np.ones((64, 3), bool)
    keep[3, 1] = keep[10, 0] = keep[40, 2] = False
    assert np.array_equal(out[0][keep], out[1][keep])
    assert not np.isfinite(out[1][3, 1]).all()
