"""Hash-sorted tables below the sizes at which the planner takes them (7 * 2^23 rows), so
that the sort, the key directory and the bucket bounds are tested where they can go
wrong: bucket groups too large for shared memory, long runs, the directory's choice
by the length of the runs, probes that take its general path."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(vals, base=0):
    return np.stack([np.arange(base, base + len(vals)), vals], 1).astype(np.int32)


@pytest.fixture()
def sorted_engine(engine):
    engine.set_option("build", native.EJ_BUILD_MSD)
    yield engine
    engine.set_option("build", 0)
    engine.set_option("partition_bits", -1)


def _check(engine, R, S, outer=False):
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    assert engine.count("hash", Rd, Sd) == len(want)
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd).cpu().numpy()), want)  # count, then write
    out = torch.full((len(want) + 8, 4), -7, dtype=torch.int32, device="cuda")
    for algo in ("hash", "single_hash", "hash_index"):
        got = engine.join(algo, Rd, Sd, out[: len(want)])
        assert np.array_equal(O.canon(got.cpu().numpy()), want), algo
        assert bool((out[len(want):] == -7).all())
    if outer:
        got = engine.join("left_outer", Rd, Sd)
        assert np.array_equal(O.canon(got.cpu().numpy()), O.canon(O.left_outer_join(R, S)))


@pytest.mark.parametrize("shape", ["three_keys", "hot_keys", "long_runs"])
def test_skewed_sort(sorted_engine, shape):
    """Buckets sorted through global memory (three keys; hot keys among unique ones) and runs
    longer than one thread's insertion sort."""
    rng = np.random.default_rng(len(shape))
    n = (1 << 20) + 333
    vals = rng.choice(1 << 30, size=n, replace=False)
    s = vals[rng.integers(n // 4, n, 200000)]
    if shape == "three_keys":
        vals, s = rng.integers(5, 8, n), np.concatenate([np.arange(4, 9), np.full(3, 1000), s])
        s[:5] = np.arange(4, 9)
        s[5:] = np.where((s[5:] >= 5) & (s[5:] < 8), 1 << 30, s[5:])
    elif shape == "hot_keys":
        vals[: n // 5] = vals[rng.integers(0, 40, n // 5)]
        s[:8] = vals[:8]
    else:
        at = 0
        for run in rng.integers(40, 3000, 60):
            vals[at: at + run] = vals[at]
            at += run
        s[:100] = vals[rng.integers(0, at, 100)]
    R = _rel(vals[rng.permutation(n)])
    _check(sorted_engine, R, _rel(s, n), outer=shape != "three_keys")


@pytest.mark.parametrize("n,dup", [((1 << 22) - 1, 3), (1 << 22, 1), (1 << 22, 3), ((1 << 23) + 5, 1)])
def test_directory_or_bounds(sorted_engine, n, dup):
    """From 2^22 rows on a sorted table keeps its directory when its runs average two rows (else the
    header's bits are 0 and it is probed through bounds)."""
    rng = np.random.default_rng(n + dup)
    keys = rng.permutation(1 << 24)[: n // dup + 1]
    R = _rel(np.repeat(keys, dup)[:n][rng.permutation(n)])
    S = _rel(np.concatenate([keys[rng.integers(0, len(keys), 300000)], rng.integers(0, 1 << 25, 100077)]), n)
    for bits in (-1, 0, 5):
        sorted_engine.set_option("partition_bits", bits)
        _check(sorted_engine, R, S, outer=bits == 0)


def test_batch_of_an_empty_and_a_small_join_beside_a_sorted_one(sorted_engine):
    """A build option reaches the joins of a batch that run as single joins, and no others."""
    rng = np.random.default_rng(3)
    sizes = [0, 500, 40000, (1 << 22) + 3]
    host = [(_rel(rng.integers(0, max(n, 1), n)), _rel(rng.integers(0, max(n, 1), 20000), 1 << 24)) for n in sizes]
    pairs = [(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()) for R, S in host]
    want = [O.canon(O.hash_join(R, S)) for R, S in host]
    outs = [torch.empty((max(len(w), 1), 4), dtype=torch.int32, device="cuda") for w in want]
    for g, w in zip(sorted_engine.batch_hash_join(pairs, outs), want):
        assert np.array_equal(O.canon(g.cpu().numpy()), w)
