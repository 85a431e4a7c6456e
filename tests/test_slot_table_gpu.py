"""Slot tables (open addressing, 16385 to 2^26 rows) where they can go wrong, in
every join that probes one, against the oracle: the hashes whose low 31 bits
are zero (no single-row form), keys of 30, 31, 32 and thousands of rows, homes
crowded at both ends of the array (long walks, wrapping round, and past the
bucket groups of the large build, above 2^21 rows), the ends of the size
range."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import JoinError
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


def _case(name, rng):
    """(R vals, S vals)"""
    if name == "special_hashes":  # alone, and with several rows
        sp = _unhash([0, 0x80000000, 1, 0x80000001, M])
        r = np.concatenate([sp, sp[1:2], rng.integers(1, 10 ** 9, 20000)])
        return r, np.concatenate([np.repeat(sp, 7), rng.integers(1, 10 ** 9, 3000), [5, -5]])
    if name == "absent_special":  # not in R: probes end at empty slots
        return rng.integers(1, 10 ** 9, 17000), np.concatenate([_unhash([0, 0x80000000]), rng.integers(1, 10 ** 9, 99)])
    if name == "run_lengths":
        r = np.concatenate([np.repeat(7, 30), np.repeat(8, 31), np.repeat(9, 32), np.repeat(10, 5000),
                            np.repeat(np.arange(100, 6100), 3)])
        return r, np.concatenate([[7, 8, 9, 9, 10, 11], rng.integers(90, 6200, 5000)])
    if name == "crowded_homes":  # thousands of keys with one home, at the array's start, middle and end
        low = rng.integers(1, 1 << 15, size=(3, 1500), dtype=np.uint64)
        h = np.concatenate([low[0], low[1] + np.uint64(0x7FFF0000), low[2] + np.uint64(0xFFFF0000)])
        v = _unhash(h)
        r = np.concatenate([v, v[:500], rng.integers(0, 10 ** 9, 15000)])
        return r, np.concatenate([v, _unhash(h ^ np.uint64(0x80000000)), _unhash(h ^ np.uint64(1))])
    assert name == "smallest"
    return np.arange(16385), rng.integers(-10, 16500, 4001)


def _rel(vals, base, rng):
    a = np.empty((len(vals), 2), dtype=np.int32)
    a[:, 0] = np.arange(base, base + len(vals))
    a[:, 1] = vals
    a[:, 1] = a[rng.permutation(len(vals)), 1]
    a[rng.integers(0, len(a)), 0] = 0  # a key of zero
    return a


@pytest.mark.parametrize("large", [False, True], ids=["direct", "grouped"])
@pytest.mark.parametrize("name", ["special_hashes", "absent_special", "run_lengths", "crowded_homes", "smallest"])
def test_slot_table(engine, name, large):
    rng = np.random.default_rng(len(name))
    rv, sv = _case(name, rng)
    if large:  # enough other rows for the build by bucket groups
        rv = np.concatenate([rv, np.arange(1100000000, 1100000000 + (1 << 21))])
        if name == "run_lengths":  # a bucket group far larger than shared memory
            rv = np.concatenate([rv, np.repeat(10, 20000)])
    R, S = _rel(rv, 0, rng), _rel(sv, 1 << 20, rng)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    inner, outer = O.canon(O.hash_join(R, S)), O.canon(O.left_outer_join(R, S))
    assert engine.count("hash", Rd, Sd) == len(inner)
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd).cpu().numpy()), inner)  # count, then write
    out = torch.empty((len(outer) + 1, 4), dtype=torch.int32, device="cuda")
    for algo in ("hash", "single_hash", "hash_index"):
        assert np.array_equal(O.canon(engine.join(algo, Rd, Sd, out).cpu().numpy()), inner), algo
    assert np.array_equal(O.canon(engine.join("left_outer", Rd, Sd, out).cpu().numpy()), outer)
    # both columns of facts over slot tables, and over one slot table and one sorted table
    F2 = _rel(np.resize(rv[:50], len(S)), 1 << 21, rng)
    D2 = _rel(np.concatenate([rv[:50], np.arange(2 * 10 ** 9, 2 * 10 ** 9 + 17000)]), 5, rng)
    want = O.canon(O.star_join3(S, F2, R, D2))
    args = [torch.from_numpy(a).cuda() for a in (S, F2, R, D2)]
    assert np.array_equal(O.canon(engine.star_join3(*args).cpu().numpy()), want)


def test_build_sizes(engine):
    """The last size of the direct build, the first built by bucket groups, and a larger one."""
    for n in (1 << 21, (1 << 21) + 1, 1 << 24):
        R = torch.empty((n, 2), dtype=torch.int32, device="cuda")
        R[:, 0] = torch.arange(n, device="cuda")
        R[:, 1] = torch.randperm(n, device="cuda") * 3
        S = torch.empty((50001, 2), dtype=torch.int32, device="cuda")
        S[:, 0] = torch.arange(50001, device="cuda")
        S[:, 1] = torch.randint(0, 3 * n, (50001,), device="cuda")
        hit = int((S[:, 1] % 3 == 0).sum())
        rows = engine.hash_join(S=S, R=R)
        assert rows.shape[0] == hit == engine.count("hash", R, S)
        assert bool((R[rows[:, 0].long(), 1] == rows[:, 1]).all()) and bool((rows[:, 1] == rows[:, 3]).all())
        assert bool((S[rows[:, 2].long(), 1] == rows[:, 3]).all()) and rows[:, 2].unique().numel() == hit


@pytest.mark.parametrize("keys", [1, 50, 3000])
def test_groups_without_rows(engine, keys):
    """More than 2^21 rows of few keys: most bucket groups of the large build are empty, others
    far larger than shared memory."""
    rng = np.random.default_rng(keys)
    n = (1 << 21) + 1000
    R = _rel(rng.integers(0, keys, n) * 7919, 0, rng)
    S = _rel(np.concatenate([np.arange(20) * 7919 % (7919 * keys), rng.integers(0, 1 << 30, 70000)]), 1 << 23, rng)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    got = engine.join("left_outer", Rd, Sd)
    assert np.array_equal(O.canon(got.cpu().numpy()), O.canon(O.left_outer_join(R, S)))
    want = O.canon(O.hash_join(R, S))
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd).cpu().numpy()), want)
    out = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd, out=out).cpu().numpy()), want)


def test_build_survives_a_scan_that_gave_up(engine):
    """With no time to wait, scans of the large build's passes give up: the joins report it or
    are right, and the same handle is right afterwards."""
    rng = np.random.default_rng(17)
    rv = np.concatenate([rng.integers(0, 1 << 20, (1 << 21) + 77), np.repeat(5, 300)])
    R, S = _rel(rv, 0, rng), _rel(rng.integers(0, 1 << 21, 100001), 1 << 23, rng)
    Rd, Sd = torch.from_numpy(R).cuda(), torch.from_numpy(S).cuda()
    want = O.canon(O.hash_join(R, S))
    out = torch.empty((len(want), 4), dtype=torch.int32, device="cuda")
    engine.set_option("wait_limit_ns", 0)
    try:
        for _ in range(3):
            try:
                got = engine.hash_join(Rd, Sd, out=out)
                assert np.array_equal(O.canon(got.cpu().numpy()), want)
            except JoinError as e:
                assert e.status == native.EJ_ERR_TIMEOUT, e
    finally:
        engine.set_option("wait_limit_ns", -1)
    assert np.array_equal(O.canon(engine.hash_join(Rd, Sd, out=out).cpu().numpy()), want)
