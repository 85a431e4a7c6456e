"""Distance joins of few S points (up to 112 in 2-D and 160 in 3-D are compared with
every R point) and of points that crowd in few cells (buckets of 256 rows and more
are shared out over the device as a list of items).  At the sizes where that begins
and where an item ends, with few and many S points, with no room left in the list,
and no slower than the same pairs with the crowd on the other side."""
import time

import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import Engine, JoinError
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
@pytest.mark.parametrize("n", [255, 256, 257, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("s", [1, 33, 112, 113, 160, 161, 700])
def test_one_crowded_cell(engine, dims, n, s):
    """A radius past all points, with and without matches, and a second crowd next to the first."""
    rng = np.random.default_rng(n * s + dims)
    rv, sv = rng.random((n, dims)), rng.random((s, dims))
    assert _check(engine, dims, rv, sv, 3.0) == n * s
    assert _check(engine, dims, rv * 0.01, sv * 0.01 + 1.2, 1.0) == 0
    both = np.concatenate([rv, rv + 4.0, rng.random((40, dims)) * 1e6])
    _check(engine, dims, both, np.concatenate([sv, sv + 3.5, [[np.nan] * dims, [np.inf] * dims]]), 1.0)


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("radius", [1.0, 1e19, 1e200, 0.0])
def test_few_points_with_odd_values(engine, dims, radius):
    """Values that never match, or only at radii whose floats overflow, on both sides of few S points."""
    rng = np.random.default_rng(8)
    odd = np.array([1e300, -1e300, 1e18, 3.5e38, 1e19, np.inf, -np.inf, np.nan, 5e-324, -0.0, 0.0, 1e150])
    rv, sv = rng.random((3000, dims)) * 2.0, rng.random((100, dims)) * 2.0
    rv[::7] = rng.choice(odd, size=rv[::7].shape)
    sv[::3] = rng.choice(odd, size=sv[::3].shape)
    _check(engine, dims, rv, sv, radius)


@pytest.mark.parametrize("dims", [2, 3])
def test_crowded_cells_of_many_points(engine, dims):
    """S points over several crowded cells, different ones in a warp."""
    rng = np.random.default_rng(dims)
    at = rng.integers(0, 3, size=(12000, dims)) * 2.0
    rv = at + rng.random(at.shape) * 0.4
    sv = rng.integers(0, 3, size=(700, dims)) * 2.0 + rng.random((700, dims)) * 0.4 - 0.3
    assert _check(engine, dims, rv, sv, 0.2) > 1000


def test_no_room_in_the_list(engine):
    """32 crowded buckets per 32 S points, more than the list holds: 256 copies of each of 4096
    sites, every S point within the radius of one site."""
    rng = np.random.default_rng(4)
    x, y = np.meshgrid(np.arange(64) * 10.0, np.arange(64) * 10.0)
    sites = np.stack([x.ravel(), y.ravel()], 1)
    n = (1 << 20) + (1 << 18) + 7
    sv = sites[rng.integers(0, 4096, n)] + rng.random((n, 2)) * 0.5
    dR = engine.points_to_device(_points(2, np.repeat(sites, 256, 0), 1))
    dS = engine.points_to_device(_points(2, sv, 1))
    assert engine.distance_join_count(dR, dS, 2, 1.0) == 256 * n


def test_buckets_in_parts_and_whole(engine):
    """One bucket of 40000 rows looked up by 90000 S points: the part of the list for buckets in
    parts fills up, the rest goes in whole."""
    rng = np.random.default_rng(6)
    dR = engine.points_to_device(_points(3, rng.random((40000, 3)) * 0.1, 1))
    dS = engine.points_to_device(_points(3, rng.random((90000, 3)) * 0.1, 1))
    assert engine.distance_join_count(dR, dS, 3, 1.0) == 40000 * 90000


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("radius", [30.0, 2000.0])
@pytest.mark.parametrize("s", [64, 150])
def test_crowd_on_either_side(engine, dims, radius, s):
    """The distance of a pair is the same both ways round, so is the count, and a crowded R with
    few S points takes no more than 20 times as long as few R points with many S points."""
    rng = np.random.default_rng(5)
    few = engine.points_to_device(_points(dims, rng.random((s, dims)) * 1000.0, 1))
    many = engine.points_to_device(_points(dims, rng.random((1 << 20, dims)) * 1000.0, 100))

    def timed(R, S):
        n = engine.distance_join_count(R, S, dims, radius)
        best = float("inf")
        for _ in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            assert engine.distance_join_count(R, S, dims, radius) == n
            best = min(best, time.perf_counter() - t)
        return n, best

    n, t = timed(many, few)
    m, u = timed(few, many)
    assert n == m > 0
    assert t < 20 * u, (t, u)


@pytest.mark.parametrize("dims", [2, 3])
def test_memory_is_short(dims):
    """R goes in smaller pieces when the scratch for all of it cannot be had (spread points and a
    crowd), the call fails only when none can."""
    rng = np.random.default_rng(7)
    rv = np.concatenate([rng.random((300000, dims)) * 300.0, rng.random((2000, dims)) * 0.5])
    sv = np.concatenate([rng.random((1000, dims)) * 300.0, rng.random((20, dims)) * 0.5])
    lib = native.load()
    with Engine(0) as e:
        try:
            lib.ej_inject_alloc_failures(2)
            assert _check(e, dims, rv, sv, 1.0) > 20 * 2000
            e.trim()
            lib.ej_inject_alloc_failures(20)
            with pytest.raises(JoinError) as x:
                _check(e, dims, rv, sv, 1.0)
            assert x.value.status == native.EJ_ERR_NOMEM
        finally:
            lib.ej_inject_alloc_failures(0)
        _check(e, dims, rv, sv, 1.0)
