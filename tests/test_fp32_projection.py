"""The FP32 formats' reunitarisation (increments from exactly summed deviations)
against the FP64 projection rounded once, on the host build of the device code."""
import numpy as np
import pytest

from tests import _hostcheck as hc

# deviations of the stored rows: rounding, a long run, the edge of the increment form, beyond it
DRIFTS = [0.0, 3e-6, 2e-4, 4e-3]


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [(4, 4, 4), (3, 3, 3), (8, 5, 2)])  # odd volume: a padded pair
@pytest.mark.parametrize("drift", DRIFTS)
def test_projection_is_the_fp64_one_rounded_once(oracle_port, nc, shape, drift):
    """Both forms round each entry once from values good to about 2e-10, so an entry
    differs by one FP32 ulp at most (6e-8 below 1) and only where the exact value lies
    within 2e-10 of the middle of two FP32 numbers: about 2e-10 / 3e-8 of the entries."""
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
    Ua, Ub = A.download()[0], B.download()[0]
    if nc == 3:  # the stored rows (row 2 is rebuilt on load): entries (i, j) at i + 3 j
        stored = [2 * (i + 3 * j) + c for i in (0, 1) for j in range(3) for c in (0, 1)]
        Ua, Ub = Ua[:, :, stored], Ub[:, :, stored]
    d = np.abs(Ua - Ub)
    assert d.max() <= 2.0 ** -24
    assert np.mean(d > 0) <= 0.02


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
    assert np.abs(out[0][keep] - out[1][keep]).max() <= 2.0 ** -23  # the partner's row 2 is rebuilt in FP32
    assert not np.isfinite(out[1][3, 1]).all()
