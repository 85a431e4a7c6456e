"""Hash and left outer joins whose build side fits in shared memory (16384 rows)
at the edges of that range, of its two block shapes (4096 rows) and of the
lookup steps, against the oracle: exact rows, counts, capacity, the
asynchronous form, and the same rows as the global-memory tables give."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import JoinError
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(rng, n, keys, base=0):
    a = np.empty((n, 2), dtype=np.int32)
    a[:, 0] = np.arange(base, base + n)
    a[:, 1] = keys[rng.integers(0, len(keys), size=n)] if n else 0
    return a


def _keys(rng, n):
    k = rng.integers(-2 ** 31, 2 ** 31 - 1, size=n, dtype=np.int64).astype(np.int32)
    k[: min(n, 3)] = [-2 ** 31, 2 ** 31 - 1, 0][: min(n, 3)]
    return k


@pytest.mark.parametrize("nR,nS,nkeys", [
    (0, 100, 1), (1, 1, 1), (1, 4097, 2), (255, 63, 300), (1000, 4001, 2000), (4096, 20000, 4096),
    (4097, 20001, 6000), (16384, 70003, 16384), (16385, 65, 9000),
    (16384, 40, 1),        # one bucket holds the whole table: steps past the buffer
    (5000, 6000, 11),      # hundreds of rows a match
    (700, 400000, 900),    # many steps per warp
])
def test_sizes(engine, nR, nS, nkeys):
    rng = np.random.default_rng(nR * 7 + nS)
    keys = _keys(rng, nkeys)
    R = _rel(rng, nR, keys)
    S = _rel(rng, nS, np.concatenate([keys, _keys(rng, nkeys)]), base=nR)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    assert engine.count("hash", Rd, Sd) == len(want)
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd).cpu().numpy()), want)
    outer = O.canon(O.left_outer_join(R, S))
    out = torch.empty((len(outer), 4), dtype=torch.int32, device="cuda")
    assert np.array_equal(O.canon(engine.join("left_outer", Rd, Sd, out).cpu().numpy()), outer)
    engine.set_option("table", 1)  # tables in global memory
    try:
        assert np.array_equal(O.canon(engine.hash_join(Rd, Sd).cpu().numpy()), want)
    finally:
        engine.set_option("table", 0)


def test_capacity_and_async(engine):
    rng = np.random.default_rng(5)
    keys = _keys(rng, 50)
    R, S = _rel(rng, 900, keys), _rel(rng, 3000, keys, base=900)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    guard = torch.full((len(want) + 1, 4), 7, dtype=torch.int32, device="cuda")
    with pytest.raises(JoinError) as e:
        engine.hash_join(Rd, Sd, out=guard[: len(want) - 1])
    assert e.value.status == native.EJ_ERR_CAPACITY
    assert bool((guard[len(want) - 1:] == 7).all())
    n = torch.zeros(1, dtype=torch.int64, device="cuda")
    engine.hash_join_async(Rd, Sd, guard[: len(want) - 1], n)
    assert engine.sync_status() == native.EJ_ERR_CAPACITY and int(n) == len(want)
    engine.hash_join_async(Rd, Sd, guard[: len(want)], n)
    assert engine.sync_status() == native.EJ_OK and int(n) == len(want)
    assert np.array_equal(O.canon(guard[: len(want)].cpu().numpy()), want)


def test_kept_count_is_dropped(engine):
    """A count kept for a large join is not taken for a small join counted after it."""
    rng = np.random.default_rng(6)
    keys = _keys(rng, 30000)
    R, S = _rel(rng, 20000, keys), _rel(rng, 50000, keys, base=20000)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    n = engine.count("hash", Rd, Sd)
    small = O.canon(O.hash_join(R[:100], S))
    assert engine.count("hash", Rd[:100], Sd) == len(small)
    out = torch.empty((n, 4), dtype=torch.int32, device="cuda")
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd, out=out).cpu().numpy()), want)
