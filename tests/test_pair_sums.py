"""The sums of all observables of FP32 lattices: a pair's components summed as in FP64 (exact FP32
sums), over the whole FP32 range."""
import numpy as np
import pytest

from tests import _hostcheck as hc


def exact(e, et, b):
    e, et, b = (x.astype(np.longdouble) for x in (e, et, b))
    return np.stack([(e * e).sum((1, 2)), ((e + et) * b).sum((1, 2)) / 4], 1), \
        np.stack([(e * e).sum((1, 2)), (np.abs(e) + np.abs(et)).__mul__(np.abs(b)).sum((1, 2)) / 4], 1)


@pytest.mark.parametrize("na", [3, 8])
# field widths: ordinary, the edges of the range of exact FP32 sums, far outside it
@pytest.mark.parametrize("width", [0.5, 1e-7, 1e-13, 1e-14, 1e-20, 1e-30, 1e14, 1e15, 3e18, 1e25, 0.0])
def test_sums_as_in_fp64(na, width):
    """Sums of at most 32 products: FP64 would be good to 2^-53 of the terms' sum each; 2^-46."""
    rng = np.random.default_rng(2)
    e, et, b = (w * rng.standard_normal((500, na, 2)).astype(np.float32) for w in (width, width, 0.3))
    e, et, b = (x.astype(np.float32) for x in (e, et, b))
    v, scale = exact(e, et, b)
    for count in (1, 25):  # pairs a thread
        o, w, m = hc.pair_sums(e, et, b, count), *(x.reshape(-1, count, 2).sum(1).astype(float) for x in (v, scale))
        assert (np.abs(o - w) <= 2.0 ** -46 * m).all()


def test_infinite_and_nan_fields():
    """As FP64 sums: infinity and NaN in their own pair only."""
    e, et, b = (np.ones((4, 8, 2), np.float32) for _ in range(3))
    e[1, 2, 0], et[2, 3, 1], e[3, 0, 0] = np.inf, -np.inf, np.nan
    o = hc.pair_sums(e, et, b)
    assert o[0].tolist() == [16.0, 8.0] and o[1].tolist() == [np.inf, np.inf]
    assert o[2].tolist() == [16.0, -np.inf] and np.isnan(o[3]).all()


@pytest.mark.parametrize("na", [3, 8])
@pytest.mark.parametrize("width", [0.5, 1e-7, 1e-13, 1e-14, 1e-30, 1e14, 1e15, 1e25, 0.0])
@pytest.mark.parametrize("cancel", [False, True])  # the six terms of a restored field's violation
def test_violation_as_in_fp64(na, width, cancel):
    """Six terms: the sum to 2^-46 of the largest, and of it squares and maxima."""
    t = (width * np.random.default_rng(3).standard_normal((500, na, 6, 2))).astype(np.float32)
    if cancel:
        t[:, :, 5] = -t[:, :, :5].sum(2)
    g = t.astype(np.longdouble).sum(2).astype(float)
    o, eps = hc.violation_sums(t), 2.0 ** -46 * np.abs(t.astype(float)).max((1, 2, 3))
    many = hc.violation_sums(t, 25)
    assert (np.abs(many[:, 0] - o[:, 0].reshape(-1, 25).sum(1)) <= 1e-14 * many[:, 0]).all()
    assert (np.abs(many[:, 1:] - o[:, 1:].reshape(-1, 25, 2).max(1)) <= 1e-14 * many[:, 1:]).all()
    assert (np.abs(o[:, 0] - (g * g).sum((1, 2))) <= 2 * eps * np.abs(g).sum((1, 2)) + 2.0 ** -46 * (g * g).sum((1, 2))).all()
    assert (np.abs(o[:, 1] - np.maximum(g.max((1, 2)), 0)) <= eps).all()
    assert (np.abs(o[:, 2] - np.abs(g).max((1, 2))) <= eps).all()


def test_zero_fields_of_broken_links():
    """0 * infinity in E.B is NaN, as in FP64; zeros alone are zero."""
    z, b = np.zeros((2, 8, 2), np.float32), np.ones((2, 8, 2), np.float32)
    b[1, 4, 0] = np.inf
    o = hc.pair_sums(z, -z, b)
    assert o[0].tolist() == [0, 0] and o[1, 0] == 0 and np.isnan(o[1, 1])


def test_infinite_and_nan_violation():
    """As FP64: maxima drop NaN, squares keep it."""
    t = np.ones((4, 8, 1, 2), np.float32)
    t[1, 2, 0, 0], t[2, 3, 0, 1], t[3, 0, 0, 0] = np.inf, -np.inf, np.nan
    o = hc.violation_sums(t)
    assert o[0].tolist() == [16, 1, 1] and o[1].tolist() == [np.inf] * 3
    assert o[2].tolist() == [np.inf, 1, np.inf] and np.isnan(o[3, 0]) and o[3, 1:].tolist() == [1, 1]


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("shape", [(4, 6, 8), (24, 20, 22)])
@pytest.mark.parametrize("width", [0.7, 1e-20, 1e22])
def test_gpu_field_energy(ctx, nc, shape, width):
    """E^2 of an FP32 lattice is the FP64 sum over its stored fields (1e-13 over 10560 sites)."""
    import topologicalcymsolver_gb300 as tcym

    lat = tcym.Lattice(ctx, nc, shape, tcym.FP32)
    lat.random_links(0.3, 1)
    lat.gaussian_efield(width, 2)
    o = lat.observables(allow_nonfinite=True)
    E = lat.download()[1].astype(np.longdouble)
    want = (E * E).sum((0, 2)) / E.shape[0]
    got = np.asarray(o.as_oracle_vector()[3:6], float)
    assert (np.abs(got - want.astype(float)) <= 1e-13 * want.astype(float)).all()
    lat.close()
