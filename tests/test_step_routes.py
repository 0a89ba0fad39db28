"""The FP64 step by tiles or by sites, whichever the lattice's extents fit: the rule, and both
routes against the oracle."""
import numpy as np
import pytest

from tests import _hostcheck as hc

# by sites: a nearly full first wave of blocks and extents the tiles fit badly; tiles: small, just
# past the wave, large
SITES = [(26, 26, 26), (33, 20, 27)]
TILES = [(8, 8, 8), (24, 24, 24), (28, 28, 28), (48, 48, 48)]


def test_rule():
    assert all(hc.by_sites(n) for n in SITES) and not any(hc.by_sites(n) for n in TILES)


def test_rule_of_the_field_update():
    """Without the exponential sites win a little more."""
    assert all(hc.by_sites(n, links=False) for n in [*SITES, (32, 32, 32)])
    assert not any(hc.by_sites(n, links=False) for n in [(8, 8, 8), (28, 28, 28), (48, 48, 48)])
    assert hc.by_sites((36, 36, 36), links=False, nc=2) and not hc.by_sites((36, 36, 36), links=False, nc=3)


def state(P, nc, shape):
    V = int(np.prod(shape))
    U, E = np.zeros((V, 3, hc.NM[nc])), np.zeros((V, 3, hc.NA[nc]))
    P.random_links(shape, U, 0.5, 3)
    P.gaussian_efield(shape, E, 0.7, 4)
    return U, E


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [SITES[0]])
def test_host_by_sites(oracle_port, nc, shape):
    """Two steps: rounding, 1e-14 of fields of order 1 each."""
    P = oracle_port[nc]
    U, E = state(P, nc, shape)
    H = hc.HostLattice(nc, "f64", shape)
    H.upload(U, E)
    H.leapfrog(0.05, 2)
    P.leapfrog(shape, U, E, 0.05, 2)
    assert max(np.abs(x - y).max() for x, y in zip(H.download(), (U, E))) < 1e-13


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [*SITES, TILES[1], (32, 32, 32)])  # the last: E alone by sites
def test_gpu_routes(ctx, oracle_port, nc, shape):
    """Leapfrog, Langevin, the flow and the two half updates on each route, 1e-12 after ten steps."""
    import topologicalcymsolver_gb300 as tcym

    P = oracle_port[nc]
    U, E = state(P, nc, shape)
    lat = tcym.Lattice(ctx, nc, shape, tcym.FP64)
    lat.upload(U, E)
    lat.leapfrog(0.05, 4)
    P.leapfrog(shape, U, E, 0.05, 4)
    lat.langevin(0.02, 1.0, 0.6, 7, 5, 4)
    P.langevin(shape, U, E, 0.02, 1.0, 0.6, 7, 5, 4)
    lat.update_e(0.03)
    P.update_e(shape, U, E, 0.03)
    lat.update_u(0.03)
    P.update_u(shape, U, E, 0.03)
    assert max(np.abs(x - y).max() for x, y in zip(lat.download(), (U, E))) < 1e-12
    lat.flow(0.02, 2)
    P.flow(shape, U, E, 0.02, 2)
    assert np.abs(lat.download()[0] - U).max() < 1e-12
    lat.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [2, 3])
# the same share by sites and by tiles in one ensemble, ragged ones, and one member alone
@pytest.mark.parametrize("shapes", [[(8, 8, 8), (13, 13, 13), (16, 16, 16), (11, 5, 7), (32, 32, 32)], [(13, 13, 13)] * 12, [(17, 17, 17)] * 20,
                                    [(26, 26, 26)], [(24, 24, 24)]])
def test_gpu_ensemble_routes(ctx, oracle_port, nc, shapes):
    """FP64 members, whatever their routes, bit for bit as the lattice alone, and against the oracle: 1e-12
    after six steps."""
    import topologicalcymsolver_gb300 as tcym

    P = oracle_port[nc]
    ens, members = tcym.Ensemble(ctx), []
    for i, shape in enumerate(shapes):
        U, E = state(P, nc, shape)
        lat, alone = (tcym.Lattice(ctx, nc, shape, tcym.FP64) for _ in range(2))
        for x in (lat, alone):
            x.upload(U, E)
        if i % 2:
            alone.langevin(0.02, 1.0, 0.6, 9, 3, 6)
        else:
            alone.leapfrog(0.05, 6)
        if i % 2:
            ens.add(lat, 0.02, tcym.DYN_LANGEVIN, 1.0, 0.6, 9, 3)
            P.langevin(shape, U, E, 0.02, 1.0, 0.6, 9, 3, 6)
        else:
            ens.add(lat, 0.05)
            P.leapfrog(shape, U, E, 0.05, 6)
        members.append((lat, alone, U, E))
    ens.step(4)
    ens.step(2)
    ens.close()
    for lat, alone, U, E in members:
        assert max(np.abs(x - y).max() for x, y in zip(lat.download(), (U, E))) < 1e-12
        assert all(np.array_equal(x, y) for x, y in zip(lat.download(), alone.download()))
        lat.close()
        alone.close()
