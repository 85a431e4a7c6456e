"""Hash tables around the largest slot tables (7 * 2^23 rows), checked on the device: unique
keys and four rows a key, counted and then written, in one pass and left outer."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LINE = 7 << 23


@pytest.mark.parametrize("n", [(1 << 25) + 1, LINE, LINE + 4])
@pytest.mark.parametrize("dup", [1, 4])
def test_largest_slot_tables(engine, n, dup):
    n -= n % dup
    g = torch.Generator(device="cuda")
    g.manual_seed(n + dup)
    R = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    R[:, 0] = torch.arange(n, device="cuda")
    R[:, 1] = torch.randperm(n, device="cuda", generator=g) // dup * 3
    S = torch.empty((100003, 2), dtype=torch.int32, device="cuda")
    S[:, 0] = torch.arange(len(S), device="cuda")
    S[:, 1] = torch.randint(0, 3 * (n // dup), (len(S),), device="cuda", generator=g)
    hit = S[:, 1] % 3 == 0
    hits = int(hit.sum())
    count = engine.count("hash", R, S)
    assert count == hits * dup
    kept = engine.hash_join(R, S, out=torch.empty((count, 4), dtype=torch.int32, device="cuda"))
    single = engine.join("single_hash", R, S, torch.empty((count, 4), dtype=torch.int32, device="cuda"))
    outer = engine.join("left_outer", R, S, torch.empty((count + len(S) - hits, 4), dtype=torch.int32, device="cuda"))
    missed = outer[:, 0] == -(1 << 31)
    assert int(missed.sum()) == len(S) - hits and not bool(hit[outer[missed][:, 2].long()].any())
    for rows in (kept, single, outer[~missed]):
        assert rows.shape[0] == count
        assert bool((R[rows[:, 0].long(), 1] == rows[:, 1]).all()) and bool((rows[:, 1] == rows[:, 3]).all())
        assert bool((S[rows[:, 2].long(), 1] == rows[:, 3]).all())
        pairs = rows[:, 2].long() * (1 << 32) + rows[:, 0].long()
        assert pairs.unique().numel() == count  # all pairs, each once
    outer = kept = single = None
