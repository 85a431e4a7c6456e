"""Handles of their own in several host threads, joining different sizes at once: a
kernel's dynamic shared memory limit belongs to the function, so a call that set
it to its own size could lower it under another thread's launch."""
import threading

import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import Engine
from eating_one_gb300.serve import PER_JOIN, Server
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _pair(rng, n, s=2000):
    R = np.stack([np.arange(n), rng.integers(0, n, n)], 1).astype(np.int32)
    S = np.stack([np.arange(s), rng.integers(0, n, s)], 1).astype(np.int32)
    return torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda(), O.canon(O.hash_join(R, S))


@pytest.mark.parametrize("sizes", [(5, 4096), (4097, 16384)])
def test_servers_at_once(sizes):
    """Two schedulers launch joins in shared memory back to back, the one small, the other large
    tables of the same kernel."""
    rng = np.random.default_rng(sizes[1])
    requests, servers = 30000, []
    pairs = [_pair(rng, n, 100) for n in sizes]
    outs = [torch.empty((len(p[2]) + 1, 4), dtype=torch.int32, device="cuda") for p in pairs]
    torch.cuda.synchronize()
    try:
        for (R, S, _), o in zip(pairs, outs):
            d = native.JoinDesc(R.data_ptr(), R.shape[0], S.data_ptr(), S.shape[0], o.data_ptr(), o.shape[0])
            servers.append((Server(PER_JOIN, lanes=4), d))

        def submit(srv, d):
            for i in range(requests):
                srv.submit(d, i)

        threads = [threading.Thread(target=submit, args=s) for s in servers]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for (srv, _), (_, _, want) in zip(servers, pairs):
            srv.drain()
            done = srv.poll(requests)
            assert len(done) == requests
            assert {(c.status, c.count) for c in done} == {(native.EJ_OK, len(want))}
    finally:
        for srv, _ in servers:
            srv.close()


def test_bucket_group_builds_at_once():
    sizes = ((1 << 21) + 1, 3 << 20, (1 << 21) + 5, 4 << 20)
    rng = np.random.default_rng(9)
    errors, threads = [], []

    def work(n, R, S, want):
        try:
            with Engine(0) as e, torch.cuda.stream(torch.cuda.Stream()):
                out = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
                for _ in range(100):
                    assert e.hash_join(R, S, out=out).shape[0] == len(want), n
                assert np.array_equal(O.canon(out.cpu().numpy()), want), n
        except Exception as x:  # noqa: BLE001 - reported by the test's own thread
            errors.append((n, x))

    for n in sizes:
        threads.append(threading.Thread(target=work, args=(n, *_pair(rng, n))))
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
