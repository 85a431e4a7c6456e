"""The block nested loop at the edges of its R blocks (16384 rows, hashed in
shared memory), its S tiles (2048 tuples) and its warp steps, against the
oracle's nested loop (exact result multisets) and the count-only mode."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(rng, n, keys, base=0):
    a = np.empty((n, 2), dtype=np.int32)
    a[:, 0] = np.arange(base, base + n)
    a[:, 1] = keys[rng.integers(0, len(keys), size=n)]
    return a


@pytest.mark.parametrize("nR,nS,nkeys", [
    (1, 2049, 2), (1023, 127, 3000), (1025, 4097, 900),
    (16384, 2048, 16384),    # one full block
    (16385, 2047, 16384),    # two uneven blocks
    (32769, 6145, 20000),    # three blocks
    (3000, 3000, 7),         # buckets of hundreds of rows: several matches per S tuple and lane
    (16384, 33, 1),          # one bucket holds the whole block
])
def test_block_edges(engine, nR, nS, nkeys):
    rng = np.random.default_rng(nR * 31 + nS)
    keys = rng.integers(-2 ** 31, 2 ** 31 - 1, size=nkeys, dtype=np.int64).astype(np.int32)
    keys[: min(nkeys, 2)] = [-2 ** 31, 2 ** 31 - 1][: min(nkeys, 2)]
    R, S = _rel(rng, nR, keys), _rel(rng, nS, keys, base=nR)
    want = O.canon(O.hash_join(R, S))
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    assert engine.count("bnl", Rd, Sd) == len(want)
    assert np.array_equal(O.canon(engine.join("bnl", Rd, Sd).cpu().numpy()), want)
