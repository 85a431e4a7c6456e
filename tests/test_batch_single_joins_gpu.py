"""Batches with joins above 2^22 rows, which run as single joins behind the batch's own
launches: rows, counts and capacity of both kinds, the asynchronous form, and no
slower than the same joins one by one."""
import time

import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import Engine, JoinError
from oracle import oracle as O

pytestmark = pytest.mark.gpu

LIMIT = 1 << 22


def _rel(vals, base=0):
    return np.stack([np.arange(base, base + len(vals)), vals], 1).astype(np.int32)


def _pairs(sizes, seed=1):
    rng = np.random.default_rng(seed)
    host = []
    for i, n in enumerate(sizes):
        dup = 1 + i % 3
        R = _rel(rng.permutation(n) // dup * 5)
        S = _rel(rng.integers(0, max(1, n // dup) * 2, 30011) * 5, 1 << 24)
        host.append((R, S))
    return host, [(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()) for R, S in host]


@pytest.mark.parametrize("sizes", [[LIMIT + 1], [300, LIMIT, LIMIT + 1, 70000], [LIMIT + 5, 2000, (1 << 23) + 1, 0]])
def test_rows_and_capacity(engine, sizes):
    host, pairs = _pairs(sizes)
    want = [O.canon(O.hash_join(R, S)) for R, S in host]
    outs = [torch.full((len(w) + 4, 4), -7, dtype=torch.int32, device="cuda") for w in want]
    with Engine(0) as e:  # a handle without scratch: the single joins grow it behind the batch
        got = e.batch_hash_join(pairs, [o[: len(w)] for o, w in zip(outs, want)])
        for g, o, w in zip(got, outs, want):
            assert np.array_equal(O.canon(g.cpu().numpy()), w)
            assert bool((o[len(w):] == -7).all())
        short = max(range(len(sizes)), key=lambda i: sizes[i])
        views = [o[: len(w) // 2] if i == short else o[: len(w)] for i, (o, w) in enumerate(zip(outs, want))]
        with pytest.raises(JoinError) as x:
            e.batch_hash_join(pairs, views)
        assert x.value.status == native.EJ_ERR_CAPACITY
        for i, w in enumerate(want):
            if i != short:
                assert np.array_equal(O.canon(views[i].cpu().numpy()), w)


def test_asynchronous(engine):
    host, pairs = _pairs([5000, LIMIT + 77, 100000], seed=2)
    want = [O.canon(O.hash_join(R, S)) for R, S in host]
    outs = [torch.empty((len(w), 4), dtype=torch.int32, device="cuda") for w in want]
    descs = (native.JoinDesc * 3)()
    for d, (R, S), o in zip(descs, pairs, outs):
        d.R, d.nR, d.S, d.nS, d.out, d.out_cap = (R.data_ptr(), R.shape[0], S.data_ptr(), S.shape[0], o.data_ptr(),
                                                  o.shape[0])
    counts = torch.zeros(3, dtype=torch.int64, device="cuda")
    engine.batch_hash_join_async(descs, 3, counts)
    assert engine.sync_status() == native.EJ_OK
    assert counts.tolist() == [len(w) for w in want]
    for o, w in zip(outs, want):
        assert np.array_equal(O.canon(o.cpu().numpy()), w)


def test_not_slower_than_alone(engine):
    n = 1 << 24
    R = torch.stack([torch.arange(n, device="cuda"), torch.randperm(n, device="cuda") // 4], 1).int()
    S = torch.stack([torch.arange(n, device="cuda"), torch.randint(0, n // 2, (n,), device="cuda")], 1).int()
    out = torch.empty((engine.count("hash", R, S), 4), dtype=torch.int32, device="cuda")

    def best(call):
        t = []
        for _ in range(7):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            call()
            t.append(time.perf_counter() - t0)
        return min(t)

    batch = best(lambda: engine.batch_hash_join([(R, S)], [out]))
    alone = best(lambda: engine.hash_join(R, S, out=out))
    assert batch < 1.25 * alone, (batch, alone)
