"""Checkerboard flow of FP32 lattices long or thin, whose tiles take other shapes than 8 x 4 x 4 pairs or
do not fit a launch."""
import numpy as np
import pytest

from tests import _hostcheck as hc


# usual shapes keep 8 x 4 x 4; None: per site (SU(2) of few sites, nz / 2 odd)
ROUTES = [((16, 16, 16), 3, (8, 4, 4)), ((20, 20, 20), 2, (8, 4, 4)), ((50, 50, 52), 2, (8, 4, 4)),
          ((96, 96, 96), 3, (8, 4, 4)), ((16, 16, 16), 2, None), ((18, 18, 18), 3, None)]
THIN = [(2, 256, 256), (4, 64, 64), (256, 2, 256), (256, 256, 4), (2, 2, 4096), (6, 64, 64)]


@pytest.mark.parametrize("shape, nc, tile", ROUTES)
def test_route(shape, nc, tile):
    assert hc.cb_tile(shape, nc) == tile


@pytest.mark.parametrize("shape", THIN + [(2, 2, 4), (6, 10, 12), (50, 2, 52)])
def test_thin_lattices(shape):
    """128 threads a block; where 8 x 4 x 4 would leave half the threads idle or more, a third fewer blocks at
    least."""
    tile, pairs = hc.cb_tile(shape, 3), (shape[0] // 2, shape[1], shape[2] // 2)
    blocks = lambda t: np.prod([-(-n // k) for n, k in zip(pairs, t)])
    assert np.prod(tile) == 128 and blocks(tile) <= blocks((8, 4, 4))
    if shape in THIN[:5]:
        assert 3 * blocks(tile) <= 2 * blocks((8, 4, 4))


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [(2, 64, 64), (4, 32, 36), (128, 2, 64), (64, 64, 4), (2, 2, 2048), (34, 18, 12), (6, 50, 20)])
def test_gpu_thin(ctx, oracle_port, nc, shape):
    """Two sweeps: FP32 links' rounding, 12 updates of entries below 1."""
    import topologicalcymsolver_gb300 as tcym

    U = np.zeros((int(np.prod(shape)), 3, hc.NM[nc]))
    oracle_port[nc].random_links(shape, U, 0.5, 9)
    lat = tcym.Lattice(ctx, nc, shape, tcym.FP32)
    lat.upload(U)
    lat.flow(0.05, 2, tcym.FLOW_CHECKERBOARD)
    oracle_port[nc].flow_checkerboard(shape, U, 0.05, 2)
    assert np.abs(lat.download()[0] - U).max() < 2e-6
    lat.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 2, 524296), (2, 262152, 4), (2, 4, 524280)])
def test_checkerboard(ctx, oracle_port, shape):
    """One sweep: FP32 links' rounding, 6 updates of entries below 1."""
    import topologicalcymsolver_gb300 as tcym

    V = int(np.prod(shape))
    U = np.zeros((V, 3, 4))
    oracle_port[2].random_links(shape, U, 0.5, 9)
    lat = tcym.Lattice(ctx, 2, shape, tcym.FP32)
    lat.upload(U)
    lat.flow(0.05, 1, tcym.FLOW_CHECKERBOARD)
    oracle_port[2].flow_checkerboard(shape, U, 0.05, 1)
    assert np.abs(lat.download()[0] - U).max() < 2e-6
    lat.close()
