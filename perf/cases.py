"""Timing cases of the sparse-product path, through the package's public entry points.

A program that differentiates sparse expressions meets a pattern once and then
re-evaluates it with new values many times. So most cases are value refills of a plan
that is kept (products, conversions, coalescing, dense blocks), and some are the first
meeting of a pattern (structure, plan and first values in one pass). The kinds:

* spgemm_refill     C = A B, values only
* btda_refill       C = B^T diag(d) A, values only
* batch_refill      many uneven B^T diag(d) A refilled together
* skewed_refill     C = A B with Zipf row lengths (a few very long rows), values only
* btda_build        C = B^T diag(d) A met for the first time: transpose, plan, values
* csc_refill        CSR -> CSC, values only
* csc_build         CSR -> CSC met for the first time: structure and values
* coalesce_refill   COO -> CSR with duplicates summed, values only
* coalesce_build    COO -> CSR met for the first time: structure and values
* blocks_csr_fill   dense blocks (a stacked_pd) times a sparse CSR, values
* blocks_ata_fill   A^T diag(d) A of dense blocks, values
* btda_dropin       C = B^T diag(d) A through the drop-in matrix handles: the caller's
                    new values are in host memory, and the result is read there

Patterns are drawn from the case's sizes and values from the seed: uniform distinct columns, N(0, 1) values and
d in [0.1, 10] (U[-1, 1] for the small C = A B), as the benchmark's configurations are.
"""
import math
import zlib

import numpy as np
import torch

from sparsediff_linalg_b200 import device as dv
from sparsediff_linalg_b200 import matrices as mx

F64 = torch.float64


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def listed():
    return [
        # one small product of the kind a single constraint gives: launch latency
        {"name": "spgemm_refill_2000", "kind": "spgemm_refill", "m": 2000, "k": 2000, "n": 2000, "per_row": 5,
         "ragged": False},
        # the chain-rule product of one large expression, re-evaluated every iteration
        {"name": "btda_refill_100k", "kind": "btda_refill", "m": 100000, "nA": 50000, "nB": 40000, "per_row": 8,
         "ragged": False},
        # all the chain-rule products of a problem, of uneven sizes, re-evaluated together
        {"name": "batch_refill_128", "kind": "batch_refill", "count": 128, "lo": 1000, "hi": 64000},
        # a product whose rows range from one entry to tens of thousands
        {"name": "skewed_refill_1M", "kind": "skewed_refill", "m": 1000000, "nnz": 20000000, "cap": 50000},
        # a new expression: its product met for the first time
        {"name": "btda_build_100k", "kind": "btda_build", "m": 100000, "nA": 50000, "nB": 40000, "per_row": 8,
         "ragged": False},
        # a large Jacobian's column form refreshed with new values
        {"name": "csc_refill_1M", "kind": "csc_refill", "m": 1000000, "n": 1000000, "per_row": 10, "ragged": False},
        # a Jacobian of odd shape converted once
        {"name": "csc_build_300k", "kind": "csc_build", "m": 300007, "n": 170003, "per_row": 9, "ragged": True},
        # a large assembled matrix re-assembled with new values
        {"name": "coalesce_refill_50M", "kind": "coalesce_refill", "m": 1000000, "n": 1000000, "unique": 35000000,
         "repeats": 15000000},
        # an assembled matrix met for the first time
        {"name": "coalesce_build_10M", "kind": "coalesce_build", "m": 400009, "n": 300007, "unique": 7000003,
         "repeats": 3000001},
        # a stacked affine map applied to a sparse Jacobian
        {"name": "blocks_csr_64", "kind": "blocks_csr_fill", "blocks": 64, "m0": 64, "n0": 256, "S_n": 100000,
         "per_col": 6, "spread": False},
        # the Hessian of a sum over dense blocks
        {"name": "blocks_ata_64", "kind": "blocks_ata_fill", "blocks": 64, "m0": 64, "n0": 256, "groups": 1},
        # one evaluation through the C API of the original library, host buffers
        {"name": "btda_dropin_100k", "kind": "btda_dropin", "m": 100000, "nA": 50000, "nB": 40000, "per_row": 8,
         "ragged": False},
    ]


_KINDS = ("spgemm_refill", "btda_refill", "batch_refill", "skewed_refill", "btda_build", "csc_refill", "csc_build",
          "coalesce_refill", "coalesce_build", "blocks_csr_fill", "blocks_ata_fill", "btda_dropin")


def draw(rng):
    def size(lo, hi):  # over the logarithm, odd and even
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(_KINDS)
    if kind == "spgemm_refill":
        return {"kind": kind, "m": size(300, 100000), "k": size(300, 100000), "n": size(300, 100000),
                "per_row": rng.randint(2, 10), "ragged": rng.random() < 0.5}
    if kind in ("btda_refill", "btda_build", "btda_dropin"):
        m = size(500, 100000)
        return {"kind": kind, "m": m, "nA": max(20, int(m * rng.uniform(0.3, 0.6))),
                "nB": max(20, int(m * rng.uniform(0.3, 0.6))), "per_row": rng.randint(3, 8),
                "ragged": rng.random() < 0.5}
    if kind == "batch_refill":
        return {"kind": kind, "count": size(4, 128), "lo": size(200, 2000), "hi": size(4000, 64000)}
    if kind == "skewed_refill":
        m = size(20000, 1000000)
        return {"kind": kind, "m": m, "nnz": 20 * m, "cap": max(200, m // 20)}
    if kind in ("csc_refill", "csc_build"):
        return {"kind": kind, "m": size(2000, 1000000), "n": size(2000, 1000000), "per_row": rng.randint(2, 10),
                "ragged": rng.random() < 0.5}
    if kind in ("coalesce_refill", "coalesce_build"):
        u = size(3000, 35000000 if kind == "coalesce_refill" else 9000000)
        side = max(100, int(u * rng.uniform(0.01, 0.05)))
        return {"kind": kind, "m": side + rng.randint(0, 99), "n": side + rng.randint(0, 99), "unique": u,
                "repeats": int(u * rng.uniform(0.1, 0.45))}
    if kind == "blocks_csr_fill":
        return {"kind": kind, "blocks": size(2, 64), "m0": rng.randint(7, 64), "n0": rng.randint(20, 256),
                "S_n": size(1000, 100000), "per_col": rng.randint(2, 8), "spread": rng.random() < 0.5}
    g = rng.choice((1, 1, 2, 4))
    return {"kind": kind, "blocks": g * size(1, 64 // g), "m0": rng.randint(9, 100), "n0": rng.randint(20, 256),
            "groups": g}


# ---------------------------------------------------------------- inputs
class _Draws:
    """The seeded generators of one state: a case's sizes fix its pattern (the expression),
    the seed its values (one evaluation of it)."""

    def __init__(self, case, seed):
        self.dev = _dev()
        self.g = torch.Generator(device=self.dev)
        self.g.manual_seed(zlib.crc32(repr(sorted((k, v) for k, v in case.items() if k != "name")).encode()))
        self.v = torch.Generator(device=self.dev)
        self.v.manual_seed(seed)

    def ints(self, hi, n):
        return torch.randint(0, hi, (n,), generator=self.g, device=self.dev)

    def normal(self, n):
        return torch.randn(n, generator=self.v, device=self.dev, dtype=F64)

    def uniform(self, n, lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=self.v, device=self.dev, dtype=F64)

    def csr(self, m, n, lens):
        """(p, i) int32 with lens[r] uniform columns in row r, distinct and ascending."""
        row = torch.repeat_interleave(torch.arange(m, device=self.dev), lens)
        nnz = row.numel()
        key = torch.sort(row * n + self.ints(n, nnz)).values
        for _ in range(30):  # redraw repeated columns
            dup = torch.zeros(nnz, dtype=torch.bool, device=self.dev)
            dup[1:] = key[1:] == key[:-1]
            nd = int(dup.sum())
            if nd == 0:
                break
            key[dup] = torch.div(key[dup], n, rounding_mode="floor") * n + self.ints(n, nd)
            key = torch.sort(key).values
        key = torch.unique_consecutive(key)
        row = torch.div(key, n, rounding_mode="floor")
        p = torch.zeros(m + 1, dtype=torch.int64, device=self.dev)
        p[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
        return p.int(), (key - row * n).int()

    def rows(self, m, n, per_row, ragged):
        k = min(per_row, n)
        if ragged:
            lens = torch.clamp(self.ints(2 * k, m), max=n)
        else:
            lens = torch.full((m,), k, device=self.dev, dtype=torch.int64)
        return self.csr(m, n, lens)

    def zipf_rows(self, m, n, nnz, cap):
        """Row lengths min(cap, ceil(s z)), z of a Zipf law of exponent 1.5, about nnz in all."""
        z = torch.floor(torch.rand(m, generator=self.g, device=self.dev, dtype=F64).clamp_(min=1e-9) ** -2.0)
        lo, hi = 1e-6, 100.0
        for _ in range(40):
            s = math.sqrt(lo * hi)
            if float(torch.clamp(torch.ceil(s * z), max=cap).sum()) > nnz:
                hi = s
            else:
                lo = s
        return self.csr(m, n, torch.clamp(torch.ceil(lo * z), max=min(cap, n)).long())


def _btda_inputs(r, c):
    Ap, Ai = r.rows(c["m"], c["nA"], c["per_row"], c["ragged"])
    Bp, Bi = r.rows(c["m"], c["nB"], c["per_row"], c["ragged"])
    return {"Ap": Ap, "Ai": Ai, "Bp": Bp, "Bi": Bi, "Ax": r.normal(Ai.numel()), "Bx": r.normal(Bi.numel()),
            "d": r.uniform(c["m"], 0.1, 10.0)}


def _batch_sizes(c):
    """Rows, columns and row length of each product of a batch: the sizes go over their
    logarithm, the row lengths over 4 .. 16."""
    out, q = [], 0.5
    for j in range(c["count"]):
        q = (q + 0.6180339887498949) % 1.0
        m = int(c["lo"] * (c["hi"] / c["lo"]) ** q)
        out.append({"m": m, "nA": max(16, m // 2), "nB": max(16, m // 2), "per_row": 4 + (j * 5) % 13,
                    "ragged": False})
    return out


def _coo_inputs(r, c):
    keys = r.ints(c["m"] * c["n"], c["unique"])
    keys = torch.cat([keys, keys[r.ints(c["unique"], c["repeats"])]])
    keys = keys[torch.randperm(keys.numel(), generator=r.g, device=r.dev)]
    rows = torch.div(keys, c["n"], rounding_mode="floor")
    return {"rows": rows.int(), "cols": (keys - rows * c["n"]).int(), "x": r.normal(keys.numel())}


def _blocks_inputs(r, c):
    """Dense blocks and S (CSR, per_col entries in every column). With `spread` every
    block takes its own n0 of S's rows, else all take the same."""
    nb, m0, n0 = c["blocks"], c["m0"], c["n0"]
    S_m = 2 * n0 if c["spread"] else n0
    Tp, Ti = r.rows(c["S_n"], S_m, c["per_col"], False)
    col = torch.repeat_interleave(torch.arange(c["S_n"], device=r.dev), (Tp[1:] - Tp[:-1]).long())
    key = torch.sort(Ti.long() * c["S_n"] + col).values
    row = torch.div(key, c["S_n"], rounding_mode="floor")
    Sp = torch.zeros(S_m + 1, dtype=torch.int64, device=r.dev)
    Sp[1:] = torch.cumsum(torch.bincount(row, minlength=S_m), 0)
    perms = []
    for _ in range(nb):
        if c["spread"]:
            perms.append(torch.sort(torch.randperm(S_m, generator=r.g, device=r.dev)[:n0]).values.int().cpu().numpy())
        else:
            perms.append(np.arange(n0, dtype=np.int32))
    return {"Sp": Sp.int().cpu().numpy(), "Si": (key - row * c["S_n"]).int().cpu().numpy(), "S_m": S_m,
            "perms": perms, "Bv": r.normal(nb * m0 * n0), "Sx": r.normal(key.numel())}


def _ata_layout(c):
    """Row and column sets of the blocks: each its own rows, the columns of its group."""
    nb, m0, n0, g = c["blocks"], c["m0"], c["n0"], c["groups"]
    rows = [np.arange(k * m0, (k + 1) * m0, dtype=np.int32) for k in range(nb)]
    cols = [np.arange((k % g) * n0, (k % g + 1) * n0, dtype=np.int32) for k in range(nb)]
    return rows, cols


def _inputs(c, seed):
    r, kind = _Draws(c, seed), c["kind"]
    if kind == "spgemm_refill":
        Ap, Ai = r.rows(c["m"], c["k"], c["per_row"], c["ragged"])
        Bp, Bi = r.rows(c["k"], c["n"], c["per_row"], c["ragged"])
        return {"Ap": Ap, "Ai": Ai, "Bp": Bp, "Bi": Bi, "Ax": r.uniform(Ai.numel(), -1, 1),
                "Bx": r.uniform(Bi.numel(), -1, 1)}
    if kind == "skewed_refill":
        Ap, Ai = r.zipf_rows(c["m"], c["m"], c["nnz"], c["cap"])
        Bp, Bi = r.zipf_rows(c["m"], c["m"], c["nnz"], c["cap"])
        return {"Ap": Ap, "Ai": Ai, "Bp": Bp, "Bi": Bi, "Ax": r.normal(Ai.numel()), "Bx": r.normal(Bi.numel())}
    if kind in ("btda_refill", "btda_build", "btda_dropin"):
        return _btda_inputs(r, c)
    if kind == "batch_refill":
        return {"parts": [_btda_inputs(r, b) for b in _batch_sizes(c)]}
    if kind in ("csc_refill", "csc_build"):
        p, i = r.rows(c["m"], c["n"], c["per_row"], c["ragged"])
        return {"p": p, "i": i, "x": r.normal(i.numel())}
    if kind in ("coalesce_refill", "coalesce_build"):
        return _coo_inputs(r, c)
    if kind == "blocks_csr_fill":
        return _blocks_inputs(r, c)
    rows, cols = _ata_layout(c)
    return {"rows": rows, "cols": cols, "X": r.normal(c["blocks"] * c["m0"] * c["n0"]),
            "d": r.uniform(c["blocks"] * c["m0"], 0.1, 10.0)}


# ---------------------------------------------------------------- the cases
def _empty(n):
    return torch.empty(max(1, n), dtype=F64, device=_dev())[:n]


class _HostView(np.ndarray):
    """A live view of a matrix handle's values that keeps the handle."""


def _kept(x, owner):
    """x, a view of memory that `owner` frees, keeping the owner with it."""
    x = x.view(_HostView) if isinstance(x, np.ndarray) else x.view(-1)
    x.owner = owner
    return x


def _host_matrix(p, i, x, m, n):
    return mx.SparseMatrix.from_csr(p.cpu().numpy(), i.cpu().numpy(), x.cpu().numpy(), m, n)


_ALIGN = 32  # doubles between the starts of a batch's outputs in their common buffer


def prepare(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    s["case"] = case
    if kind in ("spgemm_refill", "skewed_refill"):
        s["P"] = dv.Product(s["Ap"], s["Ai"], s["Bp"], s["Bi"], case.get("n", case["m"]))
        s["C"] = _empty(s["P"].nnz)
    elif kind == "btda_refill":
        s["P"], s["T"] = dv.btda_product(s["Ap"], s["Ai"], case["nA"], s["Bp"], s["Bi"], case["nB"])
        s["C"] = _empty(s["P"].nnz)
    elif kind == "batch_refill":
        prods = [dv.btda_product(q["Ap"], q["Ai"], b["nA"], q["Bp"], q["Bi"], b["nB"])[0]
                 for q, b in zip(s["parts"], _batch_sizes(case))]
        at = [0]
        for p in prods:
            at.append(at[-1] + -(-p.nnz // _ALIGN) * _ALIGN)
        s["C"] = torch.zeros(at[-1], dtype=F64, device=_dev())
        s["stream"] = torch.cuda.Stream()  # the batch is replayed from a graph, off the default stream
        s["stream"].wait_stream(torch.cuda.current_stream())
        s["batch"] = dv.Batch(prods, stream=s["stream"])
        for j, (p, q) in enumerate(zip(prods, s["parts"])):
            s["batch"].bind(j, q["Bx"], q["d"], q["Ax"], s["C"][at[j]:at[j] + p.nnz])
    elif kind == "csc_refill":
        s["T"] = dv.Transpose(s["p"], s["i"], case["m"], case["n"])
        s["C"] = _empty(s["i"].numel())
    elif kind == "coalesce_refill":
        s["K"] = dv.Coalesce(s["rows"], s["cols"], case["m"], case["n"])
        s["C"] = _empty(s["K"].nnz)
    elif kind == "blocks_csr_fill":
        nb = case["blocks"]
        s["P"] = dv.BlocksCsr([case["m0"]] * nb, [case["n0"]] * nb, s["perms"], s["Sp"], s["Si"], s["S_m"],
                              case["S_n"])
        s["C"] = _empty(s["P"].c_values)
    elif kind == "blocks_ata_fill":
        nb = case["blocks"]
        s["P"] = dv.BlocksAta([case["m0"]] * nb, [case["n0"]] * nb, s["rows"], s["cols"], nb * case["m0"],
                              case["groups"] * case["n0"])
        s["C"] = _empty(s["P"].c_values)
    elif kind == "btda_dropin":
        s["hA"], s["hB"] = s["Ax"].cpu().numpy(), s["Bx"].cpu().numpy()
        s["hd"] = s["d"].cpu().numpy()
        s["A"] = _host_matrix(s["Ap"], s["Ai"], s["Ax"], case["m"], case["nA"])
        s["B"] = _host_matrix(s["Bp"], s["Bi"], s["Bx"], case["m"], case["nB"])
        s["Cm"] = mx.BTA(s["A"], s["B"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("spgemm_refill", "skewed_refill"):
        s["P"].fill(s["Ax"], None, s["Bx"], s["C"])
        return s["C"]
    if kind == "btda_refill":
        s["P"].fill(s["Bx"], s["d"], s["Ax"], s["C"])
        return s["C"]
    if kind == "batch_refill":
        s["batch"].refill(stream=s["stream"])
        return s["C"]
    if kind == "csc_refill":
        s["T"].fill(s["x"], s["C"])
        return s["C"]
    if kind == "coalesce_refill":
        s["K"].fill(s["x"], s["C"])
        return s["C"]
    if kind == "blocks_csr_fill":
        s["P"].fill(s["Bv"], s["Sx"], s["C"])
        return s["C"]
    if kind == "blocks_ata_fill":
        s["P"].fill(s["X"], s["d"], s["C"])
        return s["C"]
    if kind == "btda_build":
        P, T = dv.btda_product(s["Ap"], s["Ai"], c["nA"], s["Bp"], s["Bi"], c["nB"])
        C = _empty(P.nnz)
        P.fill(s["Bx"], s["d"], s["Ax"], C)
        return {"p": _kept(P.Cp, (P, T)), "i": _kept(P.Ci, (P, T)), "x": C}
    if kind == "csc_build":
        T = dv.Transpose(s["p"], s["i"], c["m"], c["n"])
        x = _empty(T.nnz)
        T.fill(s["x"], x)
        return {"p": _kept(T.Tp, T), "i": _kept(T.Ti, T), "x": x}
    if kind == "coalesce_build":
        K = dv.Coalesce(s["rows"], s["cols"], c["m"], c["n"])
        x = _empty(K.nnz)
        K.fill(s["x"], x)
        return {"p": _kept(K.Cp, K), "i": _kept(K.Ci, K), "x": x}
    s["A"].set_values(s["hA"])
    s["B"].set_values(s["hB"])
    mx.BTDA_fill(s["A"], s["hd"], s["B"], s["Cm"])
    return _kept(s["Cm"].values(), (s["Cm"], s["A"], s["B"]))


# ---------------------------------------------------------------- what a pass cannot do without
def _distinct(terms, cells):
    return cells * -math.expm1(-terms / cells)


def _btda_work(c, build):
    nnz = c["m"] * c["per_row"]
    terms = nnz * c["per_row"]
    out = _distinct(terms, c["nA"] * c["nB"])
    b = 12.0 * nnz * 2 + 4.0 * (c["m"] + c["nB"]) + 8.0 * c["m"] + 8.0 * out
    if build:
        b += 4.0 * out + 4.0 * c["nB"]
    return b, 2.0 * terms + nnz


def work(c):
    kind = c["kind"]
    if kind in ("btda_refill", "btda_build", "btda_dropin"):
        b, f = _btda_work(c, kind == "btda_build")
    elif kind == "batch_refill":
        both = [_btda_work(q, False) for q in _batch_sizes(c)]
        b, f = sum(x[0] for x in both), sum(x[1] for x in both)
    elif kind == "spgemm_refill":
        nA, nB = c["m"] * min(c["per_row"], c["k"]), c["k"] * min(c["per_row"], c["n"])
        terms = nA * min(c["per_row"], c["n"])
        b = 12.0 * (nA + nB) + 4.0 * (c["m"] + c["k"]) + 8.0 * _distinct(terms, c["m"] * c["n"])
        f = 2.0 * terms
    elif kind == "skewed_refill":
        terms = c["nnz"] * (c["nnz"] / c["m"])
        b = 24.0 * c["nnz"] + 8.0 * c["m"] + 8.0 * 0.75 * terms
        f = 2.0 * terms
    elif kind in ("csc_refill", "csc_build"):
        nnz = c["m"] * min(c["per_row"], c["n"])
        b, f = 20.0 * nnz, 0.0
        if kind == "csc_build":
            b += 4.0 * nnz + 4.0 * (c["m"] + c["n"])
    elif kind in ("coalesce_refill", "coalesce_build"):
        n = c["unique"] + c["repeats"]
        out = _distinct(c["unique"], c["m"] * c["n"])
        b, f = 12.0 * n + 8.0 * out, float(n)
        if kind == "coalesce_build":
            b += 4.0 * n + 4.0 * out + 4.0 * c["m"]
    elif kind == "blocks_csr_fill":
        frac = 0.5 if c["spread"] else 1.0
        terms = c["S_n"] * c["per_col"] * frac
        cols = c["S_n"] * (1.0 - 0.5 ** c["per_col"]) if c["spread"] else c["S_n"]
        b = 8.0 * c["blocks"] * c["m0"] * (c["n0"] + cols) + 12.0 * c["S_n"] * c["per_col"]
        f = 2.0 * c["blocks"] * c["m0"] * terms
    else:
        b = 8.0 * c["blocks"] * c["m0"] * (c["n0"] + 1) + 8.0 * c["groups"] * c["n0"] ** 2
        f = 2.0 * c["blocks"] * c["m0"] * c["n0"] ** 2
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same, in plain 64-bit torch
def _expand(i, x, rowsA, Ap, Ai, Ax, n):
    """Terms of a row-wise product: the entries (row, i, x) of L against A's rows, as
    (row * n + column, value)."""
    lens = (Ap[1:] - Ap[:-1]).long()[i]
    e = torch.repeat_interleave(torch.arange(i.numel(), device=i.device), lens)
    first = torch.cumsum(lens, 0) - lens
    pos = Ap.long()[i][e] + torch.arange(e.numel(), device=i.device) - first[e]
    return rowsA[e] * n + Ai.long()[pos], x[e] * Ax[pos]


def _sum_by_key(key, val):
    k, inv = torch.unique(key, return_inverse=True)
    return k, torch.zeros(k.numel(), dtype=F64, device=key.device).index_add_(0, inv, val)


def _row_of(p):
    return torch.repeat_interleave(torch.arange(p.numel() - 1, device=p.device), (p[1:] - p[:-1]).long())


def _product(Lrow, Lk, Lx, Ap, Ai, Ax, m, n):
    """(p, i, x) of the product whose L entries are (Lrow, Lk, Lx), sorted by row; a range of rows at a time."""
    lens = (Ap[1:] - Ap[:-1]).long()[Lk]
    upto = torch.cumsum(lens, 0)
    total = int(upto[-1]) if upto.numel() else 0
    keys, vals, a = [], [], 0
    while a < Lk.numel():
        b = int(torch.searchsorted(upto, (int(upto[a - 1]) if a else 0) + 60_000_000, right=True))
        b = min(max(b, a + 1), Lk.numel())
        b = int(torch.searchsorted(Lrow, Lrow[b - 1], right=True))  # whole rows
        key, val = _expand(Lk[a:b], Lx[a:b], Lrow[a:b], Ap, Ai, Ax, n)
        k, v = _sum_by_key(key, val)
        keys.append(k)
        vals.append(v)
        a = b
    if not total:
        return torch.zeros(m + 1, dtype=torch.int32), torch.zeros(0, dtype=torch.int32), torch.zeros(0, dtype=F64)
    key, val = torch.cat(keys), torch.cat(vals)
    row = torch.div(key, n, rounding_mode="floor")
    p = torch.zeros(m + 1, dtype=torch.int64, device=key.device)
    p[1:] = torch.cumsum(torch.bincount(row, minlength=m), 0)
    return p.int(), (key - row * n).int(), val


def _btda_exact(s, nA, nB):
    order = torch.sort(s["Bi"].long(), stable=True).indices
    k = _row_of(s["Bp"])[order]
    return _product(s["Bi"].long()[order], k, s["Bx"][order] * s["d"][k], s["Ap"], s["Ai"], s["Ax"], nB, nA)


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    if kind in ("spgemm_refill", "skewed_refill"):
        return _product(_row_of(s["Ap"]), s["Ai"].long(), s["Ax"], s["Bp"], s["Bi"], s["Bx"], case["m"],
                        case.get("n", case["m"]))[2]
    if kind in ("btda_refill", "btda_dropin"):
        return _btda_exact(s, case["nA"], case["nB"])[2]
    if kind == "btda_build":
        p, i, x = _btda_exact(s, case["nA"], case["nB"])
        return {"p": p, "i": i, "x": x}
    if kind == "batch_refill":
        out = []
        for q, b in zip(s["parts"], _batch_sizes(case)):
            x = _btda_exact(q, b["nA"], b["nB"])[2]
            out.append(torch.nn.functional.pad(x, (0, -x.numel() % _ALIGN)))
        return torch.cat(out)
    if kind in ("csc_refill", "csc_build"):
        i, order = torch.sort(s["i"].long(), stable=True)
        x = s["x"][order]
        if kind == "csc_refill":
            return x
        p = torch.zeros(case["n"] + 1, dtype=torch.int64, device=i.device)
        p[1:] = torch.cumsum(torch.bincount(i, minlength=case["n"]), 0)
        return {"p": p.int(), "i": _row_of(s["p"])[order].int(), "x": x}
    if kind in ("coalesce_refill", "coalesce_build"):
        key, x = _sum_by_key(s["rows"].long() * case["n"] + s["cols"].long(), s["x"])
        if kind == "coalesce_refill":
            return x
        row = torch.div(key, case["n"], rounding_mode="floor")
        p = torch.zeros(case["m"] + 1, dtype=torch.int64, device=key.device)
        p[1:] = torch.cumsum(torch.bincount(row, minlength=case["m"]), 0)
        return {"p": p.int(), "i": (key - row * case["n"]).int(), "x": x}
    if kind == "blocks_csr_fill":
        dev = s["Sx"].device
        Sp = torch.as_tensor(s["Sp"], device=dev)
        S = torch.zeros(s["S_m"], case["S_n"], dtype=F64, device=dev)
        used = torch.zeros(s["S_m"], case["S_n"], dtype=torch.bool, device=dev)
        at = (_row_of(Sp), torch.as_tensor(s["Si"], device=dev).long())
        S[at] = s["Sx"]
        used[at] = True
        X = s["Bv"].reshape(case["blocks"], case["m0"], case["n0"])
        out = []
        for k in range(case["blocks"]):
            perm = torch.as_tensor(s["perms"][k], device=dev).long()
            cols = used[perm].any(0).nonzero().reshape(-1)
            out.append((X[k] @ S[perm][:, cols]).reshape(-1))
        return torch.cat(out)
    X = s["X"].reshape(case["blocks"], case["m0"], case["n0"])
    d = s["d"].reshape(case["blocks"], case["m0"], 1)
    g = case["groups"]
    return torch.cat([sum(X[k].T @ (d[k] * X[k]) for k in range(j, case["blocks"], g)).reshape(-1)
                      for j in range(g)])
