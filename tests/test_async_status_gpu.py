"""What one call leaves in the handle's status word says nothing about another call:
asynchronous joins after one that gave up waiting, calls on another stream, the
lanes of a server."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
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
