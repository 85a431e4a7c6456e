"""The joins whose speed is measured, each through the call a program makes.

A case is one relational join (or one batch of them) over device relations, as
the engine's users run them: count-then-write and preallocated hash joins from
the smallest to the 2^26 x 2^28 skewed one, the block nested loop, distance
joins, index builds and probes, outer and star joins, a batch of served
requests and the host-buffer join.  Row ids and join keys come from the seeded
generators of include/ej_gen.h; sizes are those of workloads.py, the served
stream (serve.py) and the tests, with odd ones between them.

Every output is a relation of whole rows.  No join promises an order of its
rows, so they are listed in word order when they are read (Rows), which is
what makes two results comparable; a program that uses them does not sort
them, so a pass does not either.  How many rows match depends on the drawn
keys: the list is filled up with rows of -1 to the most a case can have.  Rows only copy input words: there is no
computed number in them that an exact value would have to be stated for.
"""
import math
import random

import torch

from eating_one_gb300 import native
from eating_one_gb300.engine import Engine
from eating_one_gb300.workloads import EJ_GEN_PERM, EJ_GEN_UNIFORM, EJ_GEN_ZIPF, make_spec

_engine = None


def engine() -> Engine:
    """One handle for the process, as a program keeps it: its scratch stays from call to call."""
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


class Rows(list):
    """The rows of one join; reading gives their number, and all of them in word order as one
    (most, words) int64 tensor."""

    def __init__(self, rows: torch.Tensor, most: int):
        super().__init__([rows])
        self.most = most

    def __iter__(self):
        rows = list.__getitem__(self, 0)
        words = rows.contiguous().view(torch.int64)
        for w in range(words.shape[1]):
            words = words[torch.sort(words[:, w], stable=True).indices]
        whole = torch.full((max(self.most, words.shape[0]), words.shape[1]), -1, dtype=torch.int64,
                           device=words.device)
        whole[: words.shape[0]] = words
        yield words.shape[0]
        yield whole


# ---- the cases ----------------------------------------------------------------


def listed():
    return [
        # the smallest call: a lookup table of a thousand rows (the served stream's smallest
        # request, |S| = 4 |R|), the program lets the engine size the output: launches count
        {"name": "hash_1k", "kind": "hash", "r": 1000, "dup": 1, "s": 4001, "zipf": 0.0, "absent": 500, "sized": False},
        # configuration C1: an ordinary foreign-key join whose table stays in L2
        {"name": "hash_c1", "kind": "hash", "r": 1 << 20, "dup": 1, "s": 1 << 22, "zipf": 0.0, "absent": 0,
         "sized": False},
        # ragged sizes, three rows a key, skewed probes, some without a match, into a buffer the
        # program has already: one pass
        {"name": "hash_ragged", "kind": "hash", "r": 3 * 1000003, "dup": 3, "s": 24000007, "zipf": 0.75,
         "absent": 100, "sized": True},
        # the headline configuration C3: 2^26 x 2^28, four rows a key, Zipf 0.75
        {"name": "hash_c3", "kind": "hash", "r": 1 << 26, "dup": 4, "s": 1 << 28, "zipf": 0.75, "absent": 100,
         "sized": False},
        # configuration C2: the block nested loop, many-to-many
        {"name": "bnl_c2", "kind": "bnl", "r": 1 << 16, "s": 1 << 20, "domain": 1 << 16, "sized": True},
        # the reference's 2-D distance workload at its largest logged size: planted pairs among
        # points far apart
        {"name": "distance_2d", "kind": "distance", "dims": 2, "r": 1 << 19, "s": 1 << 19, "shape": "planted",
         "near": 0.1},
        # 3-D points spread over a box, about three neighbours within the radius, ragged sizes
        {"name": "distance_3d_box", "kind": "distance", "dims": 3, "r": 100003, "s": 150001, "shape": "box",
         "near": 3.0},
        # a sort index built and probed once, ragged
        {"name": "sort_index", "kind": "index", "index": "sort", "kept": False, "r": 5000011, "s": 12000017,
         "absent": 500},
        # configuration C4: the left outer join, half of S without a match
        {"name": "left_outer_c4", "kind": "left_outer", "r": 1 << 24, "s": 1 << 26, "absent": 500},
        # configuration C4: two dimensions of 2^20 rows, 2^26 facts
        {"name": "star_c4", "kind": "star", "d1": 1 << 20, "d2": 1 << 20, "f": 1 << 26},
        # requests of the served stream (configuration C5: |R| log-uniform in [2^10, 2^22], |S| = 4|R|,
        # match rates 100, 50 and 12.5 %) as one batch
        {"name": "batch_32", "kind": "batch", "joins": 32, "lo": 10.0, "hi": 22.0, "sizes": 5},
        # relations and result in pinned host memory, through the out-of-core call
        {"name": "host_join", "kind": "host", "r": 1 << 20, "s": (1 << 23) + 77, "absent": 100},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    """A size spread over the logarithm of [lo, hi]; most come out odd-sized, some are powers of two."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return 1 << max(0, n.bit_length() - 1) if rng.random() < 0.2 and n >= 2 * lo else n


def draw(rng: random.Random):
    kind = rng.choice(["hash", "hash", "hash", "bnl", "distance", "distance", "index", "left_outer", "star", "batch",
                       "host"])
    if kind == "hash":
        dup = rng.choice([1, 1, 2, 3, 4, 8])
        keys = max(1, _log(rng, 700, 1 << 25) // dup)
        s = min(1 << 27, max(1, int(keys * dup * math.exp(rng.uniform(math.log(0.5), math.log(8))))))
        return {"kind": kind, "r": keys * dup, "dup": dup, "s": s, "zipf": rng.choice([0.0, 0.0, 0.75, 1.0]),
                "absent": rng.choice([0, 100, 500]), "sized": rng.random() < 0.4}
    if kind == "bnl":
        r = _log(rng, 500, 1 << 17)
        s = _log(rng, 2000, (1 << 36) // max(r, 1 << 15))
        return {"kind": kind, "r": r, "s": s, "domain": max(64, int(r * rng.choice([0.5, 1, 1, 4]))),
                "sized": rng.random() < 0.7}
    if kind == "distance":
        shape = rng.choice(["planted", "box"])
        top = (1 << 19) if shape == "planted" else 200000
        return {"kind": kind, "dims": rng.choice([2, 3]), "r": _log(rng, 1000, top), "s": _log(rng, 1000, top),
                "shape": shape, "near": 0.1 if shape == "planted" else rng.choice([0.5, 3.0])}
    if kind == "index":
        r = _log(rng, 1000, 1 << 24)
        return {"kind": kind, "index": rng.choice(["hash", "sort"]), "kept": rng.random() < 0.5, "r": r,
                "s": _log(rng, max(1000, r // 2), min(1 << 26, 8 * r)), "absent": rng.choice([0, 500])}
    if kind == "left_outer":
        r = _log(rng, 1000, 1 << 24)
        return {"kind": kind, "r": r, "s": _log(rng, max(1000, r // 2), min(1 << 26, 8 * r)),
                "absent": rng.choice([0, 100, 500])}
    if kind == "star":
        return {"kind": kind, "d1": _log(rng, 1000, 1 << 20), "d2": _log(rng, 1000, 1 << 20),
                "f": _log(rng, 10000, 1 << 26)}
    if kind == "batch":
        return {"kind": kind, "joins": rng.randint(2, 32), "lo": 10.0, "hi": round(rng.uniform(14.0, 22.0), 2),
                "sizes": rng.randrange(1000)}
    r = _log(rng, 10000, 1 << 21)
    return {"kind": "host", "r": r, "s": _log(rng, 40000, 1 << 24), "absent": rng.choice([0, 100])}


# ---- inputs -------------------------------------------------------------------


def _r(n: int, dup: int, seed: int) -> torch.Tensor:
    """A build side: n / dup distinct keys, dup rows each, shuffled."""
    return engine().generate(make_spec(EJ_GEN_PERM, n, n // dup, 16 * seed + 1, 16 * seed + 3, dup=dup))


def _s(n: int, keys: int, seed: int, absent: int, zipf: float = 0.0) -> torch.Tensor:
    """A probe side over the build side's keys; `absent` per mille of the rows match nothing."""
    return engine().generate(make_spec(EJ_GEN_ZIPF, n, keys, 16 * seed + 2, 16 * seed + 3, absent_permille=absent,
                                       zipf_s=zipf))


def _rows(n: int, words: int = 4) -> torch.Tensor:
    return torch.empty((max(n, 1), words), dtype=torch.int32, device="cuda")


def _batch_sizes(case):
    rng = random.Random(case["sizes"])
    return [(int(2.0 ** rng.uniform(case["lo"], case["hi"])), rng.choice([1, 2, 8])) for _ in range(case["joins"])]


def _points(case, seed: int):
    """Two point relations as the engine takes them: {int32 id; double val[dims]} rows.  planted: the
    reference's generator (distinct integers below 10^9 in all dimensions, a tenth of R's values
    copied into S); box: uniform in a cube sized for `near` R points within distance 1 of a point."""
    nr, ns, dims = case["r"], case["s"], case["dims"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["shape"] == "box":
        ball = math.pi if dims == 2 else 4.0 / 3.0 * math.pi
        side = (nr * ball / case["near"]) ** (1.0 / dims)
        vals = torch.rand((nr + ns, dims), generator=g, device="cuda", dtype=torch.float64) * side
    else:
        need = nr + ns
        v = torch.unique(torch.randint(0, 10 ** 9, (need + need // 16 + 64,), generator=g, device="cuda"))
        v = v[torch.randperm(v.numel(), generator=g, device="cuda")[:need]].to(torch.float64)
        step = max(1, int(ns / (case["near"] * nr)))
        at = torch.arange(0, ns, step, device="cuda")[: min(nr, math.ceil(case["near"] * nr))]
        v[nr + at] = v[torch.randperm(nr, generator=g, device="cuda")[: at.numel()]]
        vals = v[:, None].expand(need, dims)
    words = torch.empty((nr + ns, 1 + dims), dtype=torch.int64, device="cuda")
    words[:, 0] = torch.arange(1, nr + ns + 1, device="cuda")
    words[:, 1:] = vals.contiguous().view(torch.int64)
    raw = words.view(torch.uint8)
    return raw[:nr].clone(), raw[nr:].clone()


def prepare(case, seed):
    e, kind = engine(), case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "hash":
        keys = case["r"] // case["dup"]
        st["R"] = _r(case["r"], case["dup"], seed)
        st["S"] = _s(case["s"], keys, seed, case["absent"], case["zipf"])
        st["out"] = _rows(_most(case)) if case["sized"] else None
    elif kind == "bnl":
        st["R"] = e.generate(make_spec(EJ_GEN_UNIFORM, case["r"], case["domain"], 16 * seed + 1))
        st["S"] = e.generate(make_spec(EJ_GEN_UNIFORM, case["s"], case["domain"], 16 * seed + 2))
        st["out"] = _rows(_most(case)) if case["sized"] else None
    elif kind == "distance":
        st["R"], st["S"] = _points(case, seed)
    elif kind in ("index", "left_outer"):
        st["R"] = _r(case["r"], 1, seed)
        st["S"] = _s(case["s"], case["r"], seed, case["absent"])
        st["out"] = _rows(case["s"])
        if kind == "index" and case["kept"]:
            st["index"] = e.build_index(case["index"], st["R"])
    elif kind == "star":
        st["D1"], st["D2"] = _r(case["d1"], 1, seed), _r(case["d2"], 1, seed + (1 << 40))
        st["F1"] = _s(case["f"], case["d1"], seed, 0)
        st["F2"] = _s(case["f"], case["d2"], seed + (1 << 40), 0)
        st["out"] = _rows(case["f"], 8)
    elif kind == "batch":
        st["pairs"], st["outs"] = [], []
        for i, (n, u) in enumerate(_batch_sizes(case)):
            base = (seed << 12) + i
            st["pairs"].append((e.generate(make_spec(EJ_GEN_PERM, n, n * u, 16 * base + 1, 16 * base + 3)),
                                e.generate(make_spec(EJ_GEN_UNIFORM, 4 * n, n * u, 16 * base + 2))))
            st["outs"].append(_rows(4 * n))
    else:
        host = [t.cpu().pin_memory() for t in (_r(case["r"], 1, seed), _s(case["s"], case["r"], seed, case["absent"]))]
        st["R"], st["S"] = host
        st["out"] = torch.empty((case["s"], 4), dtype=torch.int32, pin_memory=True)
    return st


def run(state):
    e, kind, case = engine(), state["kind"], state["case"]
    if kind == "batch":
        return [Rows(r, o.shape[0]) for r, o in zip(e.batch_hash_join(state["pairs"], state["outs"]), state["outs"])]
    if kind == "hash":
        rows = e.hash_join(state["R"], state["S"], state["out"])
    elif kind == "bnl":
        rows = e.join("bnl", state["R"], state["S"], state["out"])
    elif kind == "distance":
        rows = e.distance_join(state["R"], state["S"], case["dims"])
    elif kind == "index" and case["kept"]:
        rows = state["index"].join(state["S"], state["out"])
    elif kind == "index":
        ix = e.build_index(case["index"], state["R"])
        rows = ix.join(state["S"], state["out"])
        ix.free()
    elif kind == "left_outer":
        rows = e.join("left_outer", state["R"], state["S"], state["out"])
    elif kind == "star":
        rows = e.star_join3(state["F1"], state["F2"], state["D1"], state["D2"], state["out"])
    else:
        n = e.join_host_chunked("hash", state["R"], state["S"], state["out"])
        rows = state["out"][:n]
    return Rows(rows, _most(case))


# ---- what a pass cannot do without -----------------------------------------------


def _matches(case) -> float:
    """Expected result rows."""
    kind = case["kind"]
    if kind == "hash":
        return case["s"] * (1.0 - case["absent"] / 1000.0) * case["dup"]
    if kind == "bnl":
        return case["r"] * case["s"] / case["domain"]
    if kind == "distance":
        return case["s"] * case["near"] if case["shape"] == "box" else min(case["s"], case["near"] * case["r"])
    if kind == "left_outer":
        return float(case["s"])
    if kind == "star":
        return float(case["f"])
    return case["s"] * (1.0 - case["absent"] / 1000.0)


def _most(case) -> int:
    """The most result rows a program makes room for: every probe's longest run, or half as many
    again as expected where the matches are left to chance."""
    kind = case["kind"]
    if kind == "hash":
        return case["s"] * case["dup"]
    if kind in ("bnl", "distance"):
        return int(1.5 * _matches(case)) + 4096
    return case["f"] if kind == "star" else case["s"]


def work(case):
    """Every input row read once, every result row written once."""
    kind = case["kind"]
    if kind == "distance":
        pb, rb = (native.point_dtype(case["dims"]).itemsize, native.point_result_dtype(case["dims"]).itemsize)
        return {"bytes": pb * (case["r"] + case["s"]) + rb * _matches(case), "flops": 0}
    if kind == "star":
        return {"bytes": 8 * (case["d1"] + case["d2"] + 2 * case["f"]) + 32 * _matches(case), "flops": 0}
    if kind == "batch":
        return {"bytes": sum(8 * 5 * n + 16 * 4 * n / u for n, u in _batch_sizes(case)), "flops": 0}
    return {"bytes": 8 * (case["r"] + case["s"]) + 16 * _matches(case), "flops": 0}
