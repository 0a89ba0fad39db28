"""The FP32 reunitarisation of links near the identity (cooled fields), whose entries differ in
size, against the FP64 projection rounded once, bit for bit."""
import numpy as np
import pytest

from tests import _hostcheck as hc

WIDTHS = [0.3, 1e-2, 1e-4, 1e-7, 1e-20, 1e-31, 1e-40]


def links(P, nc, shape, width, drift):
    """Links of that width, of full FP32 accuracy at any: U = 1 + i x, projected, and drifted."""
    V = int(np.prod(shape))
    U = np.zeros((V, 3, hc.NM[nc]))
    if width > 1e-8:
        P.random_links(shape, U, width, 5)
    else:
        P.random_links(shape, U, 0.0, 5)  # the identity, with entries of that size beside it
        U = np.where(U == 0, width * np.random.default_rng(4).standard_normal(U.shape), U)
    return U * (1 + drift * np.random.default_rng(3).uniform(-1, 1, size=U.shape))


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("width", WIDTHS)
@pytest.mark.parametrize("drift", [0.0, 3e-7, 1.5e-5])
def test_projection_bits(oracle_port, nc, width, drift):
    shape = (16, 16, 14)
    U = links(oracle_port[nc], nc, shape, width, drift)
    A, B = hc.HostLattice(nc, "f32", shape), hc.HostLattice(nc, "f32", shape)
    for H in (A, B):
        H.upload(U, None)
    A.reunitarize()
    B.reunitarize_fp64()
    assert np.array_equal(A.download()[0], B.download()[0])


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("width", WIDTHS)
def test_gpu_projection_bits(ctx, oracle_port, nc, width):
    import topologicalcymsolver_gb300 as tcym

    shape = (16, 16, 14)
    U = links(oracle_port[nc], nc, shape, width, 3e-7)
    lat, H = tcym.Lattice(ctx, nc, shape, tcym.FP32), hc.HostLattice(nc, "f32", shape)
    lat.upload(U)
    H.upload(U, None)
    lat.reunitarize()
    H.reunitarize_fp64()
    assert np.array_equal(lat.download()[0], H.download()[0])
    lat.close()
