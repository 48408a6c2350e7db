"""The work that programs have this framework do, as cases that can be timed and compared.

Every case goes through the public entry points: batched NTTs, Poseidon2 trees, whole commitments
(alone, many in one launch, and served from host memory), query openings and the witness fill.
Elements are uniform random Goldilocks elements; all results are exact, so two correct
implementations agree in every bit.  `work` counts a modular multiplication as one operation.
"""
from __future__ import annotations

import importlib
import math
import os
import random

import numpy as np
import torch

glc = importlib.import_module("zksync-crypto-gpu_b200")

P = 0xFFFFFFFF00000001
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# any 360 field elements serve as round constants; these are installed as a prover installs boojum's
ROUND_CONSTANTS = [random.Random(360 + i).randrange(P) for i in range(360)]

_process: dict = {}


def _ready() -> None:
    """What a prover process does once: tables, round constants, the shipped launch tuning."""
    if "ctx" not in _process:
        torch.cuda.current_stream()
        _process["ctx"] = glc.Context.create()
        glc.poseidon2.set_round_constants(ROUND_CONSTANTS)
        glc.tuning.load(os.path.join(ROOT, "zksync-crypto-gpu_b200", "tuning_b200.txt"))


def _server():
    """The server of this process: programs keep one and submit to it."""
    if "server" not in _process:
        _process["server"] = glc.serve.Server(hbm_budget_bytes=40 << 30, max_inflight=16, streams=8)
    return _process["server"]


# ---- the cases ----

def listed() -> list[dict]:
    return [
        # the small configuration: one column of 2^16 to evaluations and back (launch latency)
        {"name": "roundtrip-2^16x1", "kind": "roundtrip", "log_n": 16, "cols": 1},
        # the small configuration's tree: 2^17 rows of 8 columns, cap 16
        {"name": "tree-2^17x8", "kind": "tree", "log_leaves": 17, "cols": 8, "log_rows": 0, "log_cap": 4},
        # FRI oracle: leaves of 8 rows of one extension column (2 base columns), cap 16
        {"name": "fri-2^15x2", "kind": "tree", "log_leaves": 15, "cols": 2, "log_rows": 3, "log_cap": 4},
        # smallest commitment of the uneven mix: everything is launches
        {"name": "commit-2^12x8", "kind": "commit", "log_n": 12, "cols": 8, "log_lde": 1, "log_cap": 4},
        # one coset of an LDE x4, an odd number of columns inside a wider matrix
        {"name": "coset-2^18x37", "kind": "ntt", "log_n": 18, "cols": 37, "bitrev": False, "inverse": False,
         "log_ext": 2, "coset": 3, "in_place": False, "gap": 1027},
        # evaluations of a 128-column trace to monomial form: inverse NTT and bit reversal
        {"name": "monomials-2^20x128", "kind": "monomials", "log_n": 20, "cols": 128},
        # the single-size batch configuration
        {"name": "commit-2^20x128", "kind": "commit", "log_n": 20, "cols": 128, "log_lde": 1, "log_cap": 4},
        # the large commitment: 128 base and 24 extension columns
        {"name": "commit-2^22x176", "kind": "commit", "log_n": 22, "cols": 176, "log_lde": 1, "log_cap": 4},
        # the small jobs of the uneven batch in one persistent launch
        {"name": "batch-48-uneven", "kind": "batch", "jobs": 48, "log_min": 12, "log_max": 15, "mix": 5},
        # serving: requests of uneven sizes from host memory
        {"name": "serve-8-uneven", "kind": "serve", "jobs": 8, "log_min": 14, "log_max": 17, "mix": 3},
        # query phase: 100 openings of a 2^17 x 128 coset and their Merkle paths (launch latency)
        {"name": "openings-100", "kind": "openings", "indexes": 100, "log_leaves": 17, "cols": 128, "log_cap": 3},
        # witness to trace: 2^20 rows, 150 variable and 25 witness columns, 1 of multiplicities
        {"name": "witness-2^20x176", "kind": "witness", "log_n": 20, "variables": 150, "witnesses": 25, "log_values": 26},
    ]


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["ntt", "ntt", "ntt", "monomials", "roundtrip", "tree", "tree", "commit", "commit", "batch",
                       "serve", "openings", "witness"])

    def cols_for(log_n: int, most: int = 256, elements: int = 1 << 28) -> int:
        top = max(1, min(most, elements >> log_n))
        return max(1, min(top, int(round(math.exp(rng.uniform(0.0, math.log(top + 0.49)))))))

    if kind == "ntt":
        log_n = rng.randint(1, 22) if rng.random() < 0.3 else rng.randint(10, 22)
        log_ext = rng.choice([0, 1, 2, 3])
        return {"kind": kind, "log_n": log_n, "cols": cols_for(log_n), "bitrev": rng.random() < 0.4,
                "inverse": rng.random() < 0.4, "log_ext": log_ext, "coset": rng.randrange(1 << log_ext),
                "in_place": rng.random() < 0.4, "gap": rng.choice([0, 0, 2, rng.randint(1, 999)])}
    if kind in ("monomials", "roundtrip"):
        log_n = rng.randint(10, 22)
        return {"kind": kind, "log_n": log_n, "cols": cols_for(log_n)}
    if kind == "tree":
        log_rows = rng.choice([0, 0, 0, 1, 2, 3])
        log_leaves = rng.randint(6, 21 - log_rows)
        return {"kind": kind, "log_leaves": log_leaves, "cols": cols_for(log_leaves + log_rows), "log_rows": log_rows,
                "log_cap": rng.randint(0, 5)}
    if kind == "commit":
        log_n = rng.randint(10, 21)
        log_lde = rng.choice([1, 1, 2])
        return {"kind": kind, "log_n": log_n, "cols": cols_for(log_n, elements=1 << 27), "log_lde": log_lde,
                "log_cap": rng.randint(log_lde, 6)}
    if kind == "batch":
        lo = rng.randint(12, 14)
        return {"kind": kind, "jobs": rng.randint(3, 64), "log_min": lo, "log_max": rng.randint(lo, 17),
                "mix": rng.randrange(1000)}
    if kind == "serve":
        lo = rng.randint(12, 15)
        return {"kind": kind, "jobs": rng.randint(2, 12), "log_min": lo, "log_max": rng.randint(lo, 18),
                "mix": rng.randrange(1000)}
    if kind == "openings":
        log_leaves = rng.randint(10, 20)
        return {"kind": kind, "indexes": rng.randint(1, 300), "log_leaves": log_leaves, "cols": cols_for(log_leaves),
                "log_cap": rng.randint(0, 5)}
    log_n = rng.randint(10, 21)
    return {"kind": kind, "log_n": log_n, "variables": rng.randint(1, 160), "witnesses": rng.randint(0, 40),
            "log_values": rng.randint(12, 26)}


def _mix(case: dict) -> list[tuple[int, int, int, int]]:
    """The job sizes (log_n, cols, log_lde, log_cap) of an uneven batch: the sizes follow the case, not the seed."""
    rng = random.Random(case["mix"])
    return [(rng.randint(case["log_min"], case["log_max"]), rng.choice([8, 16, 32, 64, 128]), rng.choice([1, 2]), 4)
            for _ in range(case["jobs"])]


# ---- inputs ----

def _elements(count: int, gen: torch.Generator) -> torch.Tensor:
    """Uniform field elements as the int64 bit patterns the entry points take."""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (count,), generator=gen, device="cuda", dtype=torch.int64)
    # patterns of p .. 2^64 - 1 are the int64 values -(2^32 - 1) .. -1: make them small
    chunk = 1 << 27
    for i in range(0, count, chunk):
        v = x[i:i + chunk]
        v.masked_fill_((v < 0) & (v > -(1 << 32)), 1)
    return x


def _zeros(count: int) -> torch.Tensor:
    return torch.zeros(count, dtype=torch.int64, device="cuda")


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _stride(case: dict) -> int:
    return (1 << case["log_n"]) + case.get("gap", 0)


def prepare(case: dict, seed: int) -> dict:
    _ready()
    gen = _gen(seed)
    k = case["kind"]
    st: dict = {"case": case}
    if k == "ntt":
        st["input"] = _elements(case["cols"] * _stride(case), gen)
        st["output"] = _zeros(case["cols"] * _stride(case))
    elif k in ("roundtrip", "monomials"):
        st["input"] = _elements(case["cols"] << case["log_n"], gen)
        st["output"] = _zeros(case["cols"] << case["log_n"])
        if k == "roundtrip":
            st["evals"] = _zeros(case["cols"] << case["log_n"])
    elif k == "tree":
        st["values"] = _elements(case["cols"] << (case["log_leaves"] + case["log_rows"]), gen)
        st["tree"] = _zeros(8 << case["log_leaves"])
    elif k == "commit":
        sz = glc.CommitJob.sizes(case["log_n"], case["cols"], case["log_lde"], case["log_cap"])
        st["evals"] = _elements(sz["evals"], gen)
        for name in ("monomials", "lde", "trees", "cap"):
            st[name] = _zeros(sz[name])
        st["job"] = glc.CommitJob(st["evals"], case["log_n"], case["cols"], case["log_lde"], case["log_cap"],
                                  st["lde"], st["trees"], st["cap"], monomials=st["monomials"])
    elif k == "batch":
        mix = _mix(case)
        total = {name: sum(glc.CommitJob.sizes(*m)[name] for m in mix) for name in ("evals", "lde", "trees", "cap")}
        st["evals"] = _elements(total["evals"], gen)
        for name in ("lde", "trees", "cap"):
            st[name] = _zeros(total[name])
        at = dict.fromkeys(total, 0)
        st["jobs"] = []
        for m in mix:
            part = {}
            for name, n in glc.CommitJob.sizes(*m).items():
                if name in at:
                    part[name] = st[name][at[name]:at[name] + n]
                    at[name] += n
            st["jobs"].append(glc.CommitJob(part["evals"], *m, part["lde"], part["trees"], part["cap"]))
    elif k == "serve":
        st["requests"] = []
        for m in _mix(case):
            host = torch.empty(m[1] << m[0], dtype=torch.int64, pin_memory=True)
            host.copy_(_elements(m[1] << m[0], gen))
            st["requests"].append((host.numpy().view(np.uint64), m))
        st["server"] = _server()
    elif k == "openings":
        leaves = 1 << case["log_leaves"]
        st["values"] = _elements(case["cols"] * leaves, gen)
        st["tree"] = _elements(8 * leaves, gen)
        st["indexes"] = torch.randint(0, leaves, (case["indexes"],), generator=gen, device="cuda", dtype=torch.int32)
        st["layers"] = case["log_leaves"] - case["log_cap"]
        st["rows"] = _zeros(case["indexes"] * case["cols"])
        st["paths"] = _zeros(case["indexes"] * st["layers"] * 4)
    else:
        n = 1 << case["log_n"]
        st["values"] = _elements(1 << case["log_values"], gen)

        def indexes(cols):
            i = torch.randint(0, 1 << case["log_values"], (cols * n,), generator=gen, device="cuda", dtype=torch.int32)
            hole = torch.rand(cols * n, generator=gen, device="cuda") < 0.05  # unused cells are placeholders
            return i.masked_fill_(hole, -(1 << 31))

        st["variables"] = indexes(case["variables"])
        st["witnesses"] = indexes(case["witnesses"]) if case["witnesses"] else None
        st["multiplicities"] = torch.randint(0, 1 << 20, (n - n // 3,), generator=gen, device="cuda", dtype=torch.int32)
        st["trace"] = _zeros((case["variables"] + case["witnesses"] + 1) * n)
    return st


# ---- one pass ----

def run(st: dict):
    case = st["case"]
    k = case["kind"]
    if k == "ntt":
        n, stride, out = case["log_n"], _stride(case), st["output"]
        if case["in_place"]:
            # a program that transforms in place copies what it wants to keep
            out.copy_(st["input"])
            glc.ntt.batch_ntt_in_place(out, n, case["cols"], case["gap"], stride, case["bitrev"], case["inverse"],
                                       case["log_ext"], case["coset"])
        else:
            glc.ntt.batch_ntt_out_of_place(st["input"], out, n, case["cols"], 0, case["gap"], stride, stride,
                                           case["bitrev"], case["inverse"], case["log_ext"], case["coset"])
        return out
    if k == "roundtrip":
        n, c, N = case["log_n"], case["cols"], 1 << case["log_n"]
        glc.ntt.batch_ntt_out_of_place(st["input"], st["evals"], n, c, 0, 0, N, N, False, False, 0, 0)
        glc.ntt.batch_ntt_out_of_place(st["evals"], st["output"], n, c, 0, 0, N, N, True, True, 0, 0)
        return [st["evals"], st["output"]]
    if k == "monomials":
        n, c, N = case["log_n"], case["cols"], 1 << case["log_n"]
        glc.ntt.batch_ntt_out_of_place(st["input"], st["output"], n, c, 0, 0, N, N, False, True, 0, 0)
        glc.ops_complex.bit_reverse_in_place(st["output"], N, c)
        return st["output"]
    if k == "tree":
        layers = max(1, case["log_leaves"] - case["log_cap"] + 1)
        glc.GLHasher.build_merkle_tree(st["values"], st["tree"], case["log_rows"], layers_count=layers)
        return st["tree"]
    if k == "commit":
        glc.commit.commit(st["job"])
        return [st["cap"], st["trees"], st["lde"], st["monomials"]]
    if k == "batch":
        glc.commit.commit_batch_fused(st["jobs"])
        return [st["cap"], st["trees"], st["lde"]]
    if k == "serve":
        s = st["server"]
        tickets = [s.submit(evals, *m) for evals, m in st["requests"]]
        return [s.wait(t)[0].view(np.int64) for t in tickets]
    if k == "openings":
        leaves = 1 << case["log_leaves"]
        glc.GLHasher.gather_rows(st["indexes"], 0, st["values"], leaves, case["cols"], st["rows"], case["indexes"],
                                 case["cols"])
        if st["layers"]:
            glc.GLHasher.gather_merkle_paths(st["indexes"], st["tree"], st["paths"], st["layers"])
        return [st["rows"], st["paths"]]
    glc.trace.fill_from_remote_witness_data(st["variables"], st["witnesses"], st["values"], st["multiplicities"],
                                            st["trace"], case["variables"], case["witnesses"], 1, 1 << case["log_n"])
    return st["trace"]


# ---- what a pass cannot do without ----

def _ntt_work(log_n: int, cols: int) -> tuple[int, int]:
    return 16 * cols << log_n, cols * log_n << (log_n - 1)


def _tree_work(leaves: int, per_leaf: int, cap: int) -> tuple[int, int]:
    return 8 * leaves * per_leaf + 32 * (2 * leaves - cap), 472 * (leaves * ((per_leaf + 7) // 8) + max(0, leaves - cap))


def _commit_work(log_n: int, cols: int, log_lde: int, log_cap: int, monomials: bool) -> tuple[int, int]:
    n, f = 1 << log_n, 1 << log_lde
    tree = _tree_work(f * n, cols, 1 << log_cap)
    return 8 * n * cols * (1 + f + monomials) + tree[0] - 8 * f * n * cols, (1 + f) * _ntt_work(log_n, cols)[1] + tree[1]


def work(case: dict) -> dict:
    k = case["kind"]
    if k in ("ntt", "monomials"):
        b, m = _ntt_work(case["log_n"], case["cols"])
    elif k == "roundtrip":
        b, m = (2 * x for x in _ntt_work(case["log_n"], case["cols"]))
    elif k == "tree":
        b, m = _tree_work(1 << case["log_leaves"], case["cols"] << case["log_rows"], 1 << min(case["log_leaves"], case["log_cap"]))
    elif k == "commit":
        b, m = _commit_work(case["log_n"], case["cols"], case["log_lde"], case["log_cap"], True)
    elif k in ("batch", "serve"):
        parts = [_commit_work(*j, False) for j in _mix(case)]
        b, m = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif k == "openings":
        b, m = case["indexes"] * (4 + 16 * case["cols"] + 64 * (case["log_leaves"] - case["log_cap"])), 0
    else:
        n = 1 << case["log_n"]
        b, m = (case["variables"] + case["witnesses"]) * n * 20 + n * 8 + 4 * (n - n // 3), 0
    return {"bytes": b, "flops": m}


def tolerance(case: dict):
    return "exact"


# ---- the same results from plain numpy ----

_M32, _EPS = np.uint64(0xFFFFFFFF), np.uint64(0xFFFFFFFF)
_PU = np.uint64(P)


def _canon(a):
    return np.where(a >= _PU, a - _PU, a)


def _add(a, b):
    s = a + b
    return _canon(np.where(s < a, s + _EPS, s))


def _mul(a, b):
    s32 = np.uint64(32)
    al, ah, bl, bh = a & _M32, a >> s32, b & _M32, b >> s32
    ll, lh, hl = al * bl, al * bh, ah * bl
    t = (ll >> s32) + (lh & _M32) + (hl & _M32)
    lo = (ll & _M32) | (t << s32)
    hi = ah * bh + (lh >> s32) + (hl >> s32) + (t >> s32)
    hh, h = hi >> s32, hi & _M32
    u = np.where(lo < hh, lo - hh - _EPS, lo - hh)
    v = (h << s32) - h
    r = u + v
    return _canon(np.where(r < v, r + _EPS, r))


def _powers(x: int, count: int):
    out = np.ones(1, dtype=np.uint64)
    while len(out) < count:
        out = np.concatenate([out, _mul(out, np.uint64(pow(x, len(out), P)))])
    return out[:count]


def _brev(log_n: int):
    r = np.zeros(1, dtype=np.int64)
    for _ in range(log_n):
        r = np.concatenate([2 * r, 2 * r + 1])
    return r


def _dft(x, w: int):
    """sum_j x[:, j] w^(j k) in natural order, by halving."""
    n = x.shape[1]
    if n == 1:
        return x
    e, o = _dft(x[:, 0::2], w * w % P), _dft(x[:, 1::2], w * w % P)
    o = _mul(o, _powers(w, n // 2)[None, :])
    return np.concatenate([_add(e, o), _add(e, np.where(o == 0, o, _PU - o))], axis=1)


def _ntt(x, bitrev: bool, inverse: bool, log_ext: int = 0, coset: int = 0):
    n = x.shape[1]
    log_n = n.bit_length() - 1
    w = pow(7, (P - 1) >> log_n, P)
    shift = 7 * pow(pow(7, (P - 1) >> (log_n + log_ext), P), coset, P) % P if log_ext else 1
    x = _canon(x)
    if bitrev:
        x = x[:, _brev(log_n)]
    if inverse:
        y = _mul(_dft(x, pow(w, P - 2, P)), np.uint64(pow(n, P - 2, P)))
        y = _mul(y, _powers(pow(shift, P - 2, P), n)[None, :])
    else:
        y = _dft(_mul(x, _powers(shift, n)[None, :]), w)
    return y if bitrev else y[:, _brev(log_n)]


def _external(s):
    m4 = ((5, 7, 1, 3), (4, 6, 1, 1), (1, 3, 5, 7), (1, 1, 4, 6))
    t = [[None] * 4 for _ in range(3)]
    for b in range(3):
        for i in range(4):
            acc = np.zeros_like(s[0])
            for j in range(4):
                acc = _add(acc, _mul(s[4 * b + j], np.uint64(m4[i][j])))
            t[b][i] = acc
    col = [_add(_add(t[0][i], t[1][i]), t[2][i]) for i in range(4)]
    return [_add(t[b][i], col[i]) for b in range(3) for i in range(4)]


def _permute(s):
    def sbox(x):
        x2 = _mul(x, x)
        return _mul(_mul(x2, x), _mul(x2, x2))

    rc = [np.uint64(c) for c in ROUND_CONSTANTS]
    diag = [np.uint64(1 << e) for e in (4, 14, 11, 8, 0, 5, 2, 9, 13, 6, 3, 12)]
    s = _external(s)
    for r in range(30):
        if 4 <= r < 26:
            s[0] = sbox(_add(s[0], rc[12 * r]))
            total = s[0]
            for x in s[1:]:
                total = _add(total, x)
            s = [_add(total, _mul(x, d)) for x, d in zip(s, diag)]
        else:
            s = _external([sbox(_add(x, rc[12 * r + i])) for i, x in enumerate(s)])
    return s


def _tree(values, log_rows: int, log_cap: int):
    """values (cols, leaves << log_rows) to the flat [leaf layer, node layers, unwritten tail] buffer."""
    cols, rows = values.shape
    leaves = rows >> log_rows
    flat = _canon(values).reshape(cols, leaves, 1 << log_rows).transpose(0, 2, 1).reshape(-1, leaves)
    zero = np.zeros(leaves, dtype=np.uint64)
    s = [zero] * 12
    for at in range(0, len(flat), 8):
        chunk = list(flat[at:at + 8])
        s = _permute(chunk + [zero] * (8 - len(chunk)) + s[8:])
    layer = np.stack(s[:4])
    out = [layer.reshape(-1)]
    while layer.shape[1] > (1 << log_cap):
        z = np.zeros(layer.shape[1] // 2, dtype=np.uint64)
        layer = np.stack(_permute(list(layer[:, 0::2]) + list(layer[:, 1::2]) + [z] * 4)[:4])
        out.append(layer.reshape(-1))
    flat = np.concatenate(out)
    return np.concatenate([flat, np.zeros(8 * leaves - len(flat), dtype=np.uint64)]), layer


def _signed(a):
    return np.ascontiguousarray(a).reshape(-1).view(np.int64)


def exact(case: dict, seed: int):
    k = case["kind"]
    w = work(case)
    # about 5 M modular multiplications a second
    if k in ("batch", "serve") or w["flops"] > 60_000_000 or w["bytes"] > 1 << 30:
        return None
    st = prepare(case, seed)

    def host(t):
        return t.cpu().numpy().view(np.uint64)

    if k == "ntt":
        stride, N, gap = _stride(case), 1 << case["log_n"], case["gap"]
        x = host(st["input"]).reshape(case["cols"], stride)
        off = gap if case["in_place"] else 0
        y = x.copy() if case["in_place"] else np.zeros_like(x)
        y[:, gap:gap + N] = _ntt(x[:, off:off + N], case["bitrev"], case["inverse"], case["log_ext"], case["coset"])
        return _signed(y)
    if k in ("roundtrip", "monomials"):
        x = host(st["input"]).reshape(case["cols"], -1)
        if k == "roundtrip":
            return [_signed(_ntt(x, False, False)), _signed(x)]
        return _signed(_ntt(x, False, True)[:, _brev(case["log_n"])])
    if k == "tree":
        return _signed(_tree(host(st["values"]).reshape(case["cols"], -1), case["log_rows"], case["log_cap"])[0])
    if k == "commit":
        mono = _ntt(host(st["evals"]).reshape(case["cols"], -1), False, True)[:, _brev(case["log_n"])]
        lde, trees, caps = [], [], []
        for c in range(1 << case["log_lde"]):
            lde.append(_ntt(mono, False, False, case["log_lde"], int(_brev(case["log_lde"])[c])))
            t, top = _tree(lde[-1], 0, case["log_cap"] - case["log_lde"])
            trees.append(t)
            caps.append(top)
        return [_signed(np.concatenate(caps, axis=1)), _signed(np.concatenate(trees)), _signed(np.stack(lde)), _signed(mono)]
    idx = st["indexes"].cpu().numpy().astype(np.int64) if k == "openings" else None
    if k == "openings":
        leaves = 1 << case["log_leaves"]
        rows = host(st["values"]).reshape(case["cols"], leaves)[:, idx]
        tree, paths, at = host(st["tree"]), [], 0
        for layer in range(st["layers"]):
            size = leaves >> layer
            paths.append(tree[at:at + 4 * size].reshape(4, size)[:, (idx >> layer) ^ 1])
            at += 4 * size
        return [_signed(rows), _signed(np.stack(paths)) if paths else np.zeros(0, dtype=np.int64)]
    values = host(st["values"])
    out = []
    for name in ("variables", "witnesses"):
        if st[name] is not None:
            i = st[name].cpu().numpy()
            out.append(np.where(i < 0, np.uint64(0), values[i & 0x7FFFFFFF & (len(values) - 1)]))
    n = 1 << case["log_n"]
    m = np.zeros(n, dtype=np.uint64)
    m[:n - n // 3] = st["multiplicities"].cpu().numpy().astype(np.uint64)
    return _signed(np.concatenate(out + [m]))
