"""Build sides in shared memory whose keys repeat: tuples with so many matches that the
warp writes them together (16), buckets so deep that it searches them together (128
rows), a second key in such a bucket, in the small hash and outer joins and the block
nested loop, against the oracle; and no slower than a table in global memory."""
import time

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

M = 0xFFFFFFFF


def _unhash(h):
    """The val whose 32-bit MurmurHash3 finaliser is h (uint32 arrays)."""
    h = np.asarray(h, dtype=np.uint64)
    h ^= h >> np.uint64(16)
    h = (h * np.uint64(pow(0xC2B2AE35, -1, 1 << 32))) & np.uint64(M)
    h ^= (h >> np.uint64(13)) ^ (h >> np.uint64(26))
    h = (h * np.uint64(pow(0x85EBCA6B, -1, 1 << 32))) & np.uint64(M)
    h ^= h >> np.uint64(16)
    return h.astype(np.uint32).view(np.int32)


def _rel(vals, base, rng):
    vals = np.asarray(vals)[rng.permutation(len(vals))]
    return np.stack([np.arange(base, base + len(vals)), vals], 1).astype(np.int32)


def _same(engine, R, S):
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    inner, outer = O.canon(O.hash_join(R, S)), O.canon(O.left_outer_join(R, S))
    out = torch.full((len(outer) + 8, 4), -7, dtype=torch.int32, device="cuda")
    assert engine.count("hash", Rd, Sd) == engine.count("bnl", Rd, Sd) == len(inner)
    for algo, want in (("hash", inner), ("bnl", inner), ("left_outer", outer)):
        got = engine.join(algo, Rd, Sd, out[: len(want)])
        assert np.array_equal(O.canon(got.cpu().numpy()), want), algo
        assert bool((out[len(outer):] == -7).all())


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 31, 33, 127, 128, 129, 160, 1000])
@pytest.mark.parametrize("keys", [1, 3, 13])
def test_rows_of_a_key(engine, rows, keys):
    rng = np.random.default_rng(rows * keys)
    v = rng.integers(-2 ** 31, 2 ** 31, keys)
    R = _rel(np.concatenate([np.repeat(v, rows), np.arange(1000)]), 0, rng)
    S = _rel(np.concatenate([np.resize(v, 80), np.arange(-300, 1100)]), 1 << 20, rng)
    _same(engine, R, S)


@pytest.mark.parametrize("hot", [120, 126, 129, 3000, 15000])
def test_other_keys_in_a_deep_bucket(engine, hot):
    """Keys of one bucket: a hot one, others with one, three and twenty rows, and some that only S has."""
    rng = np.random.default_rng(hot)
    v = _unhash(np.uint64(0xABCD0000) + np.arange(40, dtype=np.uint64))
    R = _rel(np.concatenate([np.repeat(v[0], hot), v[1:6], np.repeat(v[6], 3), np.repeat(v[7], 20),
                             np.arange(900)]), 0, rng)
    S = _rel(np.concatenate([v, v, v[:1], rng.integers(0, 2000, 500)]), 1 << 20, rng)
    _same(engine, R, S)


@pytest.mark.parametrize("rows,s", [(32, 1 << 22), (128, 1 << 20)])
def test_not_slower_than_a_table_in_global_memory(engine, rows, s):
    rng = np.random.default_rng(rows)
    R = torch.from_numpy(_rel(np.repeat(np.arange(16384 // rows), rows), 0, rng)).cuda()
    S = torch.from_numpy(_rel(rng.integers(0, 2 * (16384 // rows), s), 1 << 20, rng)).cuda()
    out = torch.empty((engine.count("hash", R, S), 4), dtype=torch.int32, device="cuda")

    def best():
        t = []
        for _ in range(7):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            engine.hash_join(R, S, out=out)
            t.append(time.perf_counter() - t0)
        return min(t)

    here = best()
    engine.set_option("build", 1)
    try:
        there = best()
    finally:
        engine.set_option("build", 0)
    assert here < 1.6 * there, (here, there)  # 0.7 to 1.05; lane by lane 2.1 and 2.7
