"""Options that choose a table do choose it, as options and from a tuning table."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import autotune, native
from eating_one_gb300.engine import Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(vals, base=0):
    return np.stack([np.arange(base, base + len(vals)), vals], 1).astype(np.int32)


@pytest.mark.parametrize("n", [3000, 20000, 300000, (1 << 21) + 5])
@pytest.mark.parametrize("as_option", [True, False], ids=["option", "tuning"])
def test_bucket_bounds(n, as_option):
    """A table given bucket bounds is sorted: another sequence of launches, and the same rows."""
    rng = np.random.default_rng(n)
    R, S = _rel(rng.integers(0, n, n)), _rel(rng.integers(-100, n, 70001), 1 << 23)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    out = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
    launches = []
    with Engine(0, tuned=False) as e:
        for buckets in (False, True):
            if buckets and as_option:
                e.set_option("table", native.EJ_TABLE_FORMAT_BUCKETS)
            elif buckets:
                autotune.load(e, [{"log2_rows": 0, "table": native.EJ_TABLE_FORMAT_BUCKETS}])
            before = e.kernel_launches()
            got = e.join("single_hash", Rd, Sd, out)
            launches.append(e.kernel_launches() - before)
            assert np.array_equal(O.canon(got.cpu().numpy()), want)
            for algo in ("hash", "hash_index"):
                assert np.array_equal(O.canon(e.join(algo, Rd, Sd).cpu().numpy()), want), algo
    assert launches[1] != launches[0]


@pytest.mark.parametrize("delta", [-3, 1, 2, 3])
def test_load_factor_of_a_batch(delta):
    """A bucket-bits delta of 2 or 3 makes a batch's tables emptier: more scratch, the same rows."""
    rng = np.random.default_rng(delta + 9)
    host = [(_rel(rng.integers(0, n, n)), _rel(rng.integers(-9, n, 20011), 1 << 23)) for n in (2049, 60000, 300000)]
    pairs = [(torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()) for R, S in host]
    want = [O.canon(O.hash_join(R, S)) for R, S in host]
    outs = [torch.empty((len(w), 4), dtype=torch.int32, device="cuda") for w in want]
    scratch = []
    for d in (0, delta):
        with Engine(0, tuned=False) as e:
            e.set_option("bucket_bits_delta", d)
            for g, w in zip(e.batch_hash_join(pairs, outs), want):
                assert np.array_equal(O.canon(g.cpu().numpy()), w)
            scratch.append(e.scratch_bytes())
    assert (scratch[1] > scratch[0]) == (delta > 1)
