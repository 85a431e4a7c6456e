"""The distance join's grid where it can go wrong: points on cell borders and
at exactly the radius, coordinates so large that neighbouring doubles are about
a cell apart, far outliers, one crowded cell, the warps' row buffers
overflowing - against the oracle (exact row multisets) and the count."""
import numpy as np
import pytest

from eating_one_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(dims, vals, base):
    P = np.zeros(len(vals), dtype=native.point_dtype(dims))
    P["id"] = np.arange(base, base + len(vals), dtype=np.int32)
    P["val"] = vals
    return P


def _check(engine, dims, rv, sv, radius):
    R, S = _points(dims, rv, 1), _points(dims, sv, 1 + len(rv))
    dR, dS = engine.points_to_device(R), engine.points_to_device(S)
    want = O.point_rows_canon(O.distance_join(dims, R, S, radius, threads=8))
    got = O.point_rows_canon(engine.rows_to_numpy(engine.distance_join(dR, dS, dims, radius), dims))
    assert got.shape == want.shape and np.array_equal(got, want)
    assert engine.distance_join_count(dR, dS, dims, radius) == len(want)
    return len(want)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("radius,scale", [(1.0, 6.0), (0.3, 2.0), (1e-9, 5e-9), (1e6, 9e6), (1e-150, 4e-150),
                                          (1e200, 3e200)])
def test_cell_borders(engine, dims, radius, scale):
    """Multiples of the radius moved by a few ulps, negative and positive."""
    rng = np.random.default_rng(dims)
    def draw(n):
        v = np.round((2 * rng.random((n, dims)) - 1) * scale / radius) * radius
        for _ in range(2):
            m = rng.integers(-1, 2, size=v.shape)
            v = np.where(m == 0, v, np.nextafter(v, np.where(m > 0, np.inf, -np.inf)))
        return v
    _check(engine, dims, draw(700), draw(901), radius)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("power", [48, 50, 51, 53, 60])
def test_coarse_doubles(engine, dims, power):
    """|x| of 2^power radii: neighbouring doubles are from a fraction of the radius to many radii apart."""
    rng = np.random.default_rng(power)
    at = (2.0 ** power) * np.where(rng.random(40) < 0.5, -1.0, 1.0)
    def draw(n):
        v = rng.choice(at, size=n)
        v = np.repeat(v[:, None], dims, 1)
        for _ in range(5):
            m = rng.integers(-1, 2, size=v.shape)
            v = np.where(m == 0, v, np.nextafter(v, np.where(m > 0, np.inf, -np.inf)))
        return v
    assert _check(engine, dims, draw(400), draw(500), 0.75) > 0


@pytest.mark.parametrize("dims", [2, 3])
def test_crowded_cell_and_outliers(engine, dims):
    """Most of R in one cell, S points with hundreds of matches each (row buffers run over), and
    values that never match among them."""
    rng = np.random.default_rng(9 + dims)
    rv, sv = rng.random((3000, dims)) * 0.9, rng.random((333, dims)) * 1.5
    odd = np.array([1e300, -1e300, 1e18, 3.5e38, np.inf, -np.inf, np.nan, 5e-324, -0.0, 0.0])
    rv[:40] = rng.choice(odd, size=(40, dims))
    sv[-40:] = rng.choice(odd, size=(40, dims))
    assert _check(engine, dims, rv, sv, 1.0) > 100000
