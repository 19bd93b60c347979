"""The work this framework is measured on: products, conversions, sums and sparse products of
the matrices its benchmark and tests are built from, through the package's public calls.

A case names an operation (`op`), a matrix family (`matrix`), its size and its types:

* ``mul``      y = op(A) x or Y = op(A) X into a buffer the program keeps (``k`` columns,
               column-major); with ``residual`` r = b - op(A) x, as an iterative solver forms it
* ``convert``  COO in random order -> CSR or CSC
* ``assemble`` the same conversion followed by the first product of the new matrix, as a
               program does whose matrix changes from step to step
* ``coo_sum``  A + transpose(A) of two COO matrices in random order
* ``spgemm``   A * A, CSR
* ``batch``    many products of uneven size in one replayed launch

Matrix families: ``grid`` (5-point stencil on an n = width x height grid, one coefficient per
entry), ``poisson`` (row lengths Poisson(mean), columns uniform), ``power`` (row lengths
Pareto(1.5) scaled to the mean, capped at 50,000, columns uniform), ``banded`` (half-bandwidth 3
and Poisson(8) entries off the band, for the batch).
"""
import math

import numpy as np
import torch

import __graft_entry__

gsa = __graft_entry__.load_package()
from genericsparsearrays_gb300 import batch as gsa_batch  # noqa: E402

DEV = "cuda"
DT = {"f32": torch.float32, "f64": torch.float64, "c32": torch.complex64, "c64": torch.complex128}
IT = {"i32": torch.int32, "i64": torch.int64}
SIZE = {"f32": 4, "f64": 8, "c32": 8, "c64": 16}
ISIZE = {"i32": 4, "i64": 8}
CAP = 50_000  # longest row of the power-law matrices


def listed():
    return [
        # a solver's inner product on a small system: the call's own cost
        {"name": "spmv_small", "op": "mul", "matrix": "poisson", "n": 1000, "mean": 10.0, "dtype": "f64",
         "itype": "i32", "format": "csr", "trans": "N", "k": 1, "residual": False},
        # the plain CSR SpMV of the 2048 x 2048 grid, one step of an iterative solver
        {"name": "spmv_grid", "op": "mul", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f64",
         "itype": "i32", "format": "csr", "trans": "N", "k": 1, "residual": False},
        # the same grid in single precision on a block of 16 vectors (block solvers, time steppers)
        {"name": "spmm_grid_f32", "op": "mul", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f32",
         "itype": "i32", "format": "csr", "trans": "N", "k": 16, "residual": False},
        # CSC, the layout a program that comes from SparseArrays has: the residual of a solve
        {"name": "residual_grid_csc", "op": "mul", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f64",
         "itype": "i32", "format": "csc", "trans": "N", "k": 1, "residual": True},
        # the adjoint of a random operator on a few complex vectors (least squares)
        {"name": "spmm_adjoint", "op": "mul", "matrix": "poisson", "n": 100_003, "mean": 10.0, "dtype": "c32",
         "itype": "i32", "format": "csr", "trans": "C", "k": 5, "residual": False},
        # uneven rows, complex values: graphs and Hamiltonians
        {"name": "spmv_power", "op": "mul", "matrix": "power", "n": 1_000_000, "mean": 16.0, "dtype": "c64",
         "itype": "i64", "format": "csr", "trans": "N", "k": 1, "residual": False},
        # triplets multiplied as they come, in no order
        {"name": "spmv_coo_random", "op": "mul", "matrix": "power", "n": 1_000_000, "mean": 16.0, "dtype": "c64",
         "itype": "i64", "format": "coo", "trans": "N", "k": 1, "residual": False},
        # assembled triplets of the grid to CSR
        {"name": "convert_grid", "op": "convert", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f64",
         "itype": "i64", "to": "csr"},
        # a matrix that is new in every step: triplets to CSR, then its first product
        {"name": "assemble_power", "op": "assemble", "matrix": "power", "n": 1_000_000, "mean": 16.0, "dtype": "c64",
         "itype": "i64", "to": "csr"},
        # symmetrising assembled triplets
        {"name": "coo_sum_grid", "op": "coo_sum", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f64",
         "itype": "i64"},
        # the product of a grid operator with itself (Galerkin products, polynomial filters)
        {"name": "spgemm_grid", "op": "spgemm", "matrix": "grid", "n": 2048 * 2048, "width": 2048, "dtype": "f64",
         "itype": "i32"},
        # 4096 products of uneven size, one of 1, 4 or 8 vectors each
        {"name": "batch_banded", "op": "batch", "matrix": "banded", "count": 4096, "lo": 64, "hi": 8192,
         "dtype": "c64", "itype": "i64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: products most often, as programs call them most often."""
    op = rng.choice(["mul", "mul", "mul", "mul", "convert", "assemble", "coo_sum", "spgemm", "batch"])
    dtype = rng.choice(["f32", "f64", "f64", "c32", "c64"])
    itype = rng.choice(["i32", "i64"])
    if op == "batch":
        lo = _log(rng, 32, 256)
        return {"op": op, "matrix": "banded", "count": _log(rng, 16, 4096), "lo": lo, "hi": lo * rng.choice([3, 8, 32]),
                "dtype": dtype, "itype": itype}
    family = rng.choice(["grid", "poisson", "power"])
    case = {"op": op, "matrix": family, "dtype": dtype, "itype": itype}
    if family == "grid":
        n = _log(rng, 1000, 2048 * 2048)
        width = max(2, int(math.sqrt(n) * rng.uniform(0.3, 1.4)))
        case.update(n=width * max(2, n // width), width=width)
        while case["n"] > 2048 * 2048:
            case["n"] -= width
    else:
        case.update(n=_log(rng, 1000, 1_000_000), mean=rng.choice([4.0, 7.0, 10.0, 16.0]))
    if op == "mul":
        # several FP64 columns: fewer rows, so that no case costs more than the largest listed one
        k = rng.choice([1, 1, 2, 3, 5, 8, 16])
        if case["matrix"] != "grid" and k > 8:
            k = 8
        case.update(format=rng.choice(["csr", "csr", "csc", "coo"]), trans=rng.choice(["N", "N", "T", "C"]), k=k,
                    residual=rng.random() < 0.3)
        if k > 1 and dtype in ("f64", "c64"):
            case["n"] = _shrink(case, 4)
    elif op in ("convert", "assemble"):
        case.update(to=rng.choice(["csr", "csc"]))
    elif op == "spgemm":
        # the products, not the entries, are the work: 25 a row of the grid, mean^2 of the random
        # rows, more with a power law's long rows
        if family == "grid" and dtype.startswith("c"):
            case["n"] = _shrink(case, 4)
        elif family == "poisson":
            case["mean"] = rng.choice([3.0, 4.0, 7.0, 10.0])
            case["n"] = min(case["n"], 500_000)
        elif family == "power":
            case["mean"] = rng.choice([3.0, 4.0])
            case["n"] = min(case["n"], 100_000)
    elif op == "coo_sum" and dtype == "c64":
        case["n"] = _shrink(case, 4)
    return case


def _shrink(case, by):
    n = max(1000, case["n"] // by)
    return max(2, n // case["width"]) * case["width"] if case["matrix"] == "grid" else n


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _values(count, dtype, g):
    t = DT[dtype]
    if t.is_complex:
        return torch.randn(count, 2, generator=g, device=DEV, dtype=torch.float64).view(torch.complex128)[:, 0].to(t)
    return torch.randn(count, generator=g, device=DEV, dtype=torch.float64).to(t)


def _dense(n, k, dtype, g):
    t = DT[dtype]
    if t.is_complex:
        x = _values(n * k, dtype, g)
    else:
        x = (torch.rand(n * k, generator=g, device=DEV, dtype=torch.float64) * 2 - 1).to(t)
    return x if k == 1 else x.view(k, n).t()  # column-major


def _from_lengths(lengths, n, g):
    rows = torch.repeat_interleave(torch.arange(lengths.numel(), device=DEV), lengths)
    cols = torch.randint(0, n, (rows.numel(),), generator=g, device=DEV)
    key = torch.unique(rows * n + cols)  # sorted; columns of a row distinct
    return key // n, key % n


def _structure(case, g):
    """0-based rows and columns, row by row, columns increasing; and n.  A random pattern is that
    of the case's sizes with its rows and columns renumbered from the seed: the entry counts, of
    the matrix and of its sums and products, are the same for every seed."""
    n = case["n"]
    if case["matrix"] == "grid":
        w, h = case["width"], case["n"] // case["width"]
        i = torch.arange(n, device=DEV)
        r, c = i // w, i % w
        ok = torch.stack([r > 0, c > 0, torch.ones_like(c, dtype=torch.bool), c < w - 1, r < h - 1], 1)
        cand = torch.stack([i - w, i - 1, i, i + 1, i + w], 1)
        return i[:, None].expand_as(cand)[ok], cand[ok], n
    fixed = _gen(n)
    if case["matrix"] == "poisson":
        lengths = torch.poisson(torch.full((n,), float(case["mean"]), device=DEV), generator=fixed).long()
    else:
        u = 1.0 - torch.rand(n, generator=fixed, device=DEV, dtype=torch.float64)
        lengths = torch.ceil(case["mean"] / 3.0 * u ** (-1.0 / 1.5)).clamp(max=min(CAP, max(1, n // 4))).long()
    rows, cols = _from_lengths(lengths, n, fixed)
    number = torch.randperm(n, generator=g, device=DEV)
    key = torch.sort(number[rows] * n + number[cols])[0]
    return key // n, key % n, n


def _pointers(major, n):
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(major, minlength=n), 0)
    return ptr


def _inputs(case, seed):
    """rows, cols (0-based, row by row), n and the values."""
    g = _gen(seed)
    rows, cols, n = _structure(case, g)
    return rows, cols, n, _values(rows.numel(), case["dtype"], g), g


def _shuffled(rows, cols, g):
    p = torch.randperm(rows.numel(), generator=g, device=DEV)
    return rows[p], cols[p]


def _csr(rows, cols, n, vals, it):
    return gsa.GenericSparseMatrixCSR(n, n, (_pointers(rows, n) + 1).to(it), (cols + 1).to(it), vals)


def _coo(rows, cols, n, vals, it):
    return gsa.GenericSparseMatrixCOO(n, n, (rows + 1).to(it), (cols + 1).to(it), vals)


def _matrix(case, rows, cols, n, vals, g):
    it = IT[case["itype"]]
    if case["format"] == "csr":
        return _csr(rows, cols, n, vals, it)
    if case["format"] == "coo":
        return _coo(*_shuffled(rows, cols, g), n, vals, it)
    order = torch.argsort(cols * n + rows)
    return gsa.GenericSparseMatrixCSC(n, n, (_pointers(cols, n) + 1).to(it), (rows[order] + 1).to(it), vals[order])


def _batch_parts(case, seed):
    """The batch's matrices as one block-diagonal pattern (sizes of the case, patterns of the
    seed): their sizes and first rows, columns of the dense operands, global rows, columns inside
    the matrix, values, the matrix of every row, and the generator."""
    g = _gen(seed)
    u = torch.rand(case["count"], generator=_gen(case["count"]), device=DEV, dtype=torch.float64)
    sizes = torch.exp(math.log(case["lo"]) + u * math.log(case["hi"] / case["lo"])).round().long()
    mat = torch.repeat_interleave(torch.arange(case["count"], device=DEV), sizes)  # matrix of a row
    total = mat.numel()
    first = torch.cumsum(sizes, 0) - sizes
    row = torch.arange(total, device=DEV)
    local, size = row - first[mat], sizes[mat]
    band = local[:, None] + torch.arange(-3, 4, device=DEV)
    ok = (band >= 0) & (band < size[:, None])
    extra = torch.poisson(torch.full((total,), 8.0, device=DEV), generator=g).long()
    erow = torch.repeat_interleave(row, extra)
    ecol = (torch.rand(erow.numel(), generator=g, device=DEV) * size[erow]).long().clamp(max=size[erow] - 1)
    hi = int(sizes.max())
    key = torch.unique(torch.cat([row[:, None].expand_as(band)[ok] * hi + band[ok], erow * hi + ecol]))
    rows, cols = key // hi, key % hi
    ks = [(1, 4, 8)[i % 3] for i in range(case["count"])]
    return sizes, first, ks, rows, cols, _values(rows.numel(), case["dtype"], g), mat, g


def _batch_dense(case, sizes, ks, g):
    span = [n * k for n, k in zip(sizes.tolist(), ks)]
    off = np.concatenate([[0], np.cumsum(span)]).tolist()
    return _dense(off[-1], 1, case["dtype"], g), off


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        sizes, first, ks, rows, cols, vals, _, g = _batch_parts(case, seed)
        x, off = _batch_dense(case, sizes, ks, g)
        y = torch.zeros_like(x)
        ptr = _pointers(rows, int(sizes.sum()))
        it = IT[case["itype"]]
        ends = ptr[torch.cat([first, first[-1:] + sizes[-1:]])].tolist()
        idx = (cols + 1).to(it)
        products = []
        for i, (n, r0) in enumerate(zip(sizes.tolist(), first.tolist())):
            e0, e1 = ends[i], ends[i + 1]
            A = gsa.GenericSparseMatrixCSR(n, n, (ptr[r0:r0 + n + 1] - e0 + 1).to(it), idx[e0:e1], vals[e0:e1])
            view = (lambda t: t[off[i]:off[i + 1]] if ks[i] == 1 else t[off[i]:off[i + 1]].view(ks[i], n).t())
            products.append((A, view(x), view(y), 1, 0))
        return {"op": op, "batch": gsa_batch.BatchedMul(products), "y": y}
    rows, cols, n, vals, g = _inputs(case, seed)
    it = IT[case["itype"]]
    if op == "mul":
        A = _matrix(case, rows, cols, n, vals, g)
        opA = {"N": lambda M: M, "T": gsa.transpose, "C": gsa.adjoint}[case["trans"]](A)
        x = _dense(n, case["k"], case["dtype"], g)
        y = torch.zeros_like(x)
        return {"op": op, "A": opA, "x": x, "y": y, "b": _dense(n, case["k"], case["dtype"], g)
                if case["residual"] else None}
    if op in ("convert", "assemble"):
        x = _dense(n, 1, case["dtype"], g)
        to = gsa.GenericSparseMatrixCSR if case["to"] == "csr" else gsa.GenericSparseMatrixCSC
        return {"op": op, "A": _coo(*_shuffled(rows, cols, g), n, vals, it), "to": to, "x": x}
    if op == "coo_sum":
        A = _coo(*_shuffled(rows, cols, g), n, vals, it)
        return {"op": op, "A": A, "B": gsa.transpose(A)}
    A = _csr(rows, cols, n, vals, it)
    return {"op": op, "A": A, "B": A}  # spgemm


# ---------------------------------------------------------------------------
# one pass

def _arrays(M):
    if isinstance(M, gsa.GenericSparseMatrixCSR):
        return [M.rowptr, M.colval, M.nzval]
    if isinstance(M, gsa.GenericSparseMatrixCSC):
        return [M.colptr, M.rowval, M.nzval]
    return [M.rowind, M.colind, M.nzval]


def run(state):
    op = state["op"]
    if op == "mul":
        if state["b"] is not None:
            state["y"].copy_(state["b"])
            return gsa.mul_(state["y"], state["A"], state["x"], -1, 1)
        return gsa.mul_(state["y"], state["A"], state["x"])
    if op == "convert":
        return _arrays(state["to"](state["A"]))
    if op == "assemble":
        M = state["to"](state["A"])
        return _arrays(M) + [gsa.mul(M, state["x"])]
    if op == "batch":
        state["batch"].run("graph")
        return state["y"]
    if op == "spgemm":
        return _arrays(state["A"] @ state["B"])
    return _arrays(state["A"] + state["B"])


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _entries(case):
    n = case["n"]
    if case["matrix"] == "grid":
        w, h = case["width"], n // case["width"]
        return 5 * n - 2 * w - 2 * h
    if case["matrix"] == "power":
        # E[min(cap, ceil(x_m u^(-2/3)))], half an entry for the ceiling
        cap, xm = min(CAP, max(1, n // 4)), case["mean"] / 3.0
        return n * (3 * xm - 2 * xm ** 1.5 * cap ** -0.5 + 0.5)
    return n * case["mean"]


def work(case):
    op, v, i = case["op"], SIZE[case["dtype"]], ISIZE[case["itype"]]
    mac = 8 if case["dtype"].startswith("c") else 2
    if op == "batch":
        # n log-uniform in [lo, hi]; about 15 entries a row; 13/3 columns on average
        n = case["count"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": n * (15 * (v + i) + i + 2 * 13 / 3 * v), "flops": n * 15 * 13 / 3 * mac}
    n, e = case["n"], _entries(case)
    if op == "mul":
        k = case["k"]
        a = e * (v + 2 * i) if case["format"] == "coo" else e * (v + i) + (n + 1) * i
        return {"bytes": a + n * k * v * (3 if case["residual"] else 2), "flops": e * k * mac}
    if op in ("convert", "assemble"):
        b = e * (v + 2 * i) + e * (v + i) + (n + 1) * i
        return {"bytes": b + (2 * n * v if op == "assemble" else 0), "flops": e * mac if op == "assemble" else 0}
    if op == "coo_sum":
        # the two terms share the grid's pattern; random patterns hardly overlap
        out = e if case["matrix"] == "grid" else 2 * e
        return {"bytes": e * (v + 2 * i) + out * (v + 2 * i), "flops": 0}
    # spgemm: 13 positions and 25 products a row of the grid; random patterns hardly collide
    products = 25 * n if case["matrix"] == "grid" else e * e / n
    out = 13 * n if case["matrix"] == "grid" else products
    return {"bytes": (e + out) * (v + i) + 2 * (n + 1) * i, "flops": products * mac}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch

def _wide(t):
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _sum_by_key(key, val):
    """Sorted distinct keys and their sums."""
    keys, inv = torch.unique(key, return_inverse=True)
    return keys, torch.zeros(keys.numel(), dtype=val.dtype, device=DEV).index_add_(0, inv, val)


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        sizes, first, ks, rows, cols, vals, mat, g = _batch_parts(case, seed)
        x, off = _batch_dense(case, sizes, ks, g)
        x, vals = _wide(x), _wide(vals)
        y = torch.zeros_like(x)
        off = torch.tensor(off[:-1], device=DEV)
        kk = torch.tensor(ks, device=DEV)
        m = mat[rows]
        for c in range(max(ks)):
            on = kk[m] > c
            me = m[on]
            at = off[me] + c * sizes[me]
            y.index_add_(0, at + rows[on] - first[me], vals[on] * x[at + cols[on]])
        return y
    rows, cols, n, vals, g = _inputs(case, seed)
    wide = _wide(vals)
    if op == "mul":
        vw = wide
        if case["format"] == "coo":
            rows, cols = _shuffled(rows, cols, g)
        if case["trans"] != "N":
            rows, cols = cols, rows
            vw = vw.conj().resolve_conj() if case["trans"] == "C" and vw.is_complex() else vw
        x = _wide(_dense(n, case["k"], case["dtype"], g)).reshape(n, case["k"])
        y = torch.zeros(n, case["k"], dtype=x.dtype, device=DEV)
        for c in range(case["k"]):
            y[:, c].index_add_(0, rows, vw * x[cols, c])
        y = y[:, 0] if case["k"] == 1 else y
        if case["residual"]:
            y = _wide(_dense(n, case["k"], case["dtype"], g)) - y
        return y
    if op in ("convert", "assemble"):
        x = _wide(_dense(n, 1, case["dtype"], g))
        r, c = _shuffled(rows, cols, g)
        out = [None, None, wide[torch.argsort(r * n + c if case["to"] == "csr" else c * n + r)]]
        if op == "assemble":
            out.append(torch.zeros_like(x).index_add_(0, r, wide * x[c]))
        return out
    if op == "coo_sum":
        r, c = _shuffled(rows, cols, g)
        return [None, None, _sum_by_key(torch.cat([c * n + r, r * n + c]), torch.cat([wide, wide]))[1]]
    ptr = _pointers(rows, n)
    q0 = ptr[cols]
    length = ptr[cols + 1] - q0
    t = torch.repeat_interleave(torch.arange(rows.numel(), device=DEV), length)
    q = torch.arange(t.numel(), device=DEV) - (torch.cumsum(length, 0) - length)[t] + q0[t]
    return [None, None, _sum_by_key(rows[t] * n + cols[q], wide[t] * wide[q])[1]]
