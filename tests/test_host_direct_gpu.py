"""Host-buffer hash joins whose probes read the pinned S and write the pinned out in
one pass, and the ones next to them that do not (S not 16-byte aligned,
partitioned probes), against the oracle: chunk and warp-tile edges, long runs,
every table form, a capacity one short."""
import numpy as np
import pytest
import torch

from eating_one_gb300 import native
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _pinned(a, shift=0):
    """a in pinned memory, `shift` rows behind a 16-byte boundary"""
    t = torch.empty((len(a) + shift, a.shape[1]), dtype=torch.int32).pin_memory()
    t[shift:] = torch.from_numpy(a)
    return t[shift:]


def _relations(n_r, n_s, seed):
    rng = np.random.default_rng(seed)
    R = np.stack([rng.permutation(n_r), rng.integers(-n_r // 2, n_r, n_r)], 1).astype(np.int32)
    S = np.stack([np.arange(n_s) + n_r, rng.integers(-n_r // 2, 2 * n_r, n_s)], 1).astype(np.int32)
    R[: n_r // 50, 1] = 7  # one long run
    S[::97, 1] = 7
    return R, S


@pytest.mark.parametrize("n_s", [1, 127, 128, 129, 1023, 1025, 40001])
@pytest.mark.parametrize("s_chunk", [0, 128, 1001])
@pytest.mark.parametrize("shift", [0, 1])
def test_chunks(engine, n_s, s_chunk, shift):
    R, S = _relations(3001, n_s, n_s + s_chunk)
    want = O.canon(O.hash_join(R, S))
    for r_block in (0, 1000):
        out = torch.full((len(want) + 3, 4), -1, dtype=torch.int32).pin_memory()
        n = engine.join_host_chunked("hash", _pinned(R), _pinned(S, shift), out, r_block, s_chunk)
        assert n == len(want)
        assert np.array_equal(O.canon(out[:n].numpy()), want)
        assert (out[n:] == -1).all()


@pytest.mark.parametrize("options", [{}, {"table": native.EJ_TABLE_FORMAT_DIRECTORY}, {"build": native.EJ_BUILD_LSD},
                                     {"partition_bits": 5}, {"probe_warps": 4}], ids=str)
def test_tables_and_capacity(engine, options):
    R, S = _relations(50021, 200003, 5)
    want = O.canon(O.hash_join(R, S))
    for k, v in options.items():
        engine.set_option(k, v)
    try:
        out = torch.empty((len(want), 4), dtype=torch.int32).pin_memory()
        assert engine.join_host_chunked("hash", _pinned(R), _pinned(S), out) == len(want)
        assert np.array_equal(O.canon(out.numpy()), want)
        short = torch.full((len(want), 4), -1, dtype=torch.int32).pin_memory()
        # past the capacity rows are counted, not written
        assert engine.join_host_chunked("hash", _pinned(R), _pinned(S), short[:-1]) == len(want)
        both = np.unique(np.concatenate([want, short[:-1].numpy()]), axis=0)
        assert len(both) == len(np.unique(want, axis=0)) and (short[:-1] != -1).any(dim=1).all()
        assert (short[-1] == -1).all()
    finally:
        for k in options:
            engine.set_option(k, -1 if k == "partition_bits" else 0)
