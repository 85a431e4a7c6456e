"""What one call leaves in the handle's status word says nothing about another call:
asynchronous joins after one that gave up waiting, calls on another stream, the
lanes of a server."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import JoinError
from eating_one_gb300.serve import BATCHED, PER_JOIN, Server
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(vals, base=0):
    return np.stack([np.arange(base, base + len(vals)), vals], 1).astype(np.int32)


@pytest.mark.parametrize("n", [(1 << 21) + 4097, 3 << 20])
def test_join_after_an_asynchronous_join_that_gave_up(engine, n):
    """Tables built by bucket groups stay empty when a scan of their own build gave up, not
    when an earlier call's did and nobody has read the status since."""
    rng = np.random.default_rng(n)
    R = _rel(rng.integers(0, n, n))
    S = _rel(rng.integers(0, n, 50001), 1 << 23)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    first = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
    second = torch.empty_like(first)
    counts = torch.zeros(2, dtype=torch.int64, device="cuda")
    timed_out = False
    for _ in range(10):
        engine.set_option("wait_limit_ns", 0)
        try:
            engine.hash_join_async(Rd, Sd, first, counts[:1])
        finally:
            engine.set_option("wait_limit_ns", -1)
        second.fill_(-1)
        engine.hash_join_async(Rd, Sd, second, counts[1:])
        status = engine.sync_status()
        assert status in (native.EJ_OK, native.EJ_ERR_TIMEOUT)
        timed_out |= status == native.EJ_ERR_TIMEOUT
        assert int(counts[1]) == len(want)
        assert np.array_equal(O.canon(second.cpu().numpy()), want)
    assert timed_out
    assert engine.sync_status() == native.EJ_OK


def _serve(srv, d, k):
    """Request d k times; the completions in order of their tags."""
    for i in range(k):
        srv.submit(d, i)
    srv.drain()
    return sorted(srv.poll(k), key=lambda c: c.tag)


def test_server_reports_a_request_that_gave_up(engine):
    """A lane's kernels that gave up waiting fail their own request, and no later one."""
    rng = np.random.default_rng(11)
    n = (1 << 21) + 4097
    R, S = _rel(rng.integers(0, n, n)), _rel(rng.integers(0, n, 50001), 1 << 23)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    out = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()  # the lanes have streams of their own
    d = native.JoinDesc(Rd.data_ptr(), n, Sd.data_ptr(), len(S), out.data_ptr(), len(want))
    srv = Server(PER_JOIN, lanes=1)
    try:
        srv.set_option("wait_limit_ns", 0)
        gave_up = 0
        for _ in range(10):
            c = _serve(srv, d, 1)[0]
            assert c.status in (native.EJ_OK, native.EJ_ERR_TIMEOUT)
            gave_up += c.status == native.EJ_ERR_TIMEOUT
            if c.status == native.EJ_OK:
                assert c.count == len(want)
        assert gave_up
        srv.set_option("wait_limit_ns", -1)
        for c in _serve(srv, d, 3):
            assert c.status == native.EJ_OK and c.count == len(want)
        assert np.array_equal(O.canon(out.cpu().numpy()), want)
    finally:
        srv.close()


def test_server_options_wait_for_the_requests(engine):
    """An option is refused while a request is under way, and an unknown value as by a handle."""
    rng = np.random.default_rng(12)
    R, S = _rel(rng.integers(0, 1 << 20, 1 << 20)), _rel(rng.integers(0, 1 << 20, 1 << 22), 1 << 23)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    out = torch.empty((1 << 23, 4), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    d = native.JoinDesc(Rd.data_ptr(), len(R), Sd.data_ptr(), len(S), out.data_ptr(), out.shape[0])
    srv = Server(BATCHED, lanes=1, max_batch_joins=1)
    try:
        for i in range(50):
            srv.submit(d, i)
        with pytest.raises(JoinError) as e:
            srv.set_option("partition_bits", 4)
        assert e.value.status == native.EJ_ERR_BUSY
        srv.drain()
        srv.set_option("partition_bits", 4)
        with pytest.raises(JoinError) as e:
            srv.set_option("partition_bits", 9)
        assert e.value.status == native.EJ_ERR_INVALID
        n = {c.count for c in srv.poll(100) + _serve(srv, d, 1)}
        assert n == {engine.count("hash", Rd, Sd)}
    finally:
        srv.close()


def test_status_is_clear_when_a_call_returns(engine):
    """A call that found a short capacity returns with the status word cleared and nothing of its
    own under way: the next call may use another stream, which nothing orders behind this one."""
    rng = np.random.default_rng(13)
    R, S = _rel(rng.integers(0, 1000, 3000)), _rel(rng.integers(0, 1000, 5000), 1 << 23)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    rows = len(O.left_outer_join(R, S))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    pending = 0
    for _ in range(50):
        with torch.cuda.stream(a):
            n = engine.count("left_outer", Rd, Sd)
            pending += not a.query()
        assert n == rows
        with torch.cuda.stream(b):
            engine._sync_stream()
            assert engine.sync_status() == native.EJ_OK
    assert pending == 0
