"""mul_'s short way for the usual call against its general code: the same results, bit for bit, over
formats, operations, layouts, strides, column counts, empty sizes and scalar types, and the same
errors, whichever of the two takes the call."""
import itertools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def layouts(t):
    """The matrix (n, k) in every layout a caller may hold it in."""
    n, k = t.shape
    yield "column-major", t.t().contiguous().t()
    yield "row-major", t.contiguous()
    wide = torch.zeros((k, n + 3), dtype=t.dtype, device=t.device).t()
    wide[:n].copy_(t)
    yield "padded", wide[:n]
    far = torch.zeros((n, 2 * k + 1), dtype=t.dtype, device=t.device)
    far[:, ::2][:, :k].copy_(t)
    yield "no unit stride", far[:, ::2][:, :k]
    if k == 1:
        yield "vector", t[:, 0].contiguous()
        yield "strided vector", far[:, 0]


@pytest.mark.parametrize("dt", [torch.int64, torch.float64, torch.complex128, torch.float32])
@pytest.mark.parametrize("fmt", ["csr", "csc", "coo", "coo_sorted"])
@pytest.mark.parametrize("m,n,nnz", [(40, 30, 300), (500, 700, 9000), (5, 0, 0), (0, 4, 0), (6, 7, 0), (1, 9, 4)])
def test_same_as_general(gsa, cuda, monkeypatch, fmt, dt, m, n, nnz):
    import genericsparsearrays_gb300.sparse as sparse
    plain = sparse._mul_plain
    taken = []
    rng = np.random.default_rng(nnz)
    r, c = rng.integers(0, max(m, 1), nnz), rng.integers(0, max(n, 1), nnz)
    if nnz > 1000:
        r[:800] = 3  # a row of more than a chunk
    v = torch.from_numpy(rng.integers(-4, 5, nnz)).to(dt)
    order = np.argsort(c if fmt == "csc" else r, kind="stable") if fmt != "coo" else np.arange(nnz)
    r, c = r[order] + 1, c[order] + 1
    if fmt in ("csr", "csc"):
        maj, mn, cnt = (r, c, m) if fmt == "csr" else (c, r, n)
        ptr = np.concatenate([[0], np.cumsum(np.bincount(maj - 1, minlength=cnt))]) + 1
        cls = gsa.GenericSparseMatrixCSR if fmt == "csr" else gsa.GenericSparseMatrixCSC
        A = cls(m, n, ptr, mn, v)
    else:
        A = gsa.GenericSparseMatrixCOO(m, n, r, c, v)
    A = gsa.adapt(cuda, A)
    scalars = [(1, 0), (2, 3), (-1, 1), (True, 0), (2.0, -0.0)]
    if dt.is_complex:
        scalars.append((1 + 2j, 3))
    for op, k in itertools.product("NTC", (0, 1, 2, 5)):
        M = {"N": A, "T": gsa.transpose(A), "C": gsa.adjoint(A)}[op]
        rows, inner = (m, n) if op == "N" else (n, m)
        X = torch.from_numpy(rng.integers(-4, 5, (inner, k))).to(dt).to(cuda)
        Y = torch.from_numpy(rng.integers(-4, 5, (rows, k))).to(dt).to(cuda)
        for (nx, B), (ny, C), (al, be) in itertools.product(layouts(X), layouts(Y), scalars):
            if (B.dim(), C.dim()) not in ((1, 1), (2, 2)):
                continue
            got = []
            for way in (plain, lambda *a: False, plain):  # the first may only make the plan
                monkeypatch.setattr(sparse, "_mul_plain", lambda *a, way=way: taken.append(way(*a)) or taken[-1])
                D = torch.empty_strided(C.shape, C.stride(), dtype=dt, device=cuda).copy_(C)
                got.append(gsa.mul_(D, M, B, al, be).cpu())
            assert torch.equal(got[1], got[2]), (op, k, nx, ny, al, be)
    assert any(taken) and not all(taken)


def test_same_errors(gsa, cuda, monkeypatch):
    import genericsparsearrays_gb300.sparse as sparse
    plain = sparse._mul_plain
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(2, 3, np.array([1, 2, 3]), np.array([1, 3]), np.ones(2)))
    x, y = torch.ones(3, dtype=torch.float64, device=cuda), torch.zeros(2, dtype=torch.float64, device=cuda)
    gsa.mul_(y, A, x)  # the plan is made
    calls = [(y, A, x[:2]), (x, A, x), (y, A, x.cpu()), (y.cpu(), A, x), (y, A, x.float()), (y, A, x, 1j), (y, A, 3),
             (3, A, x), (y, x, x), (y.to(torch.complex128), A, x), (y, A, torch.ones(3, 2, device=cuda).double()),
             (y.long(), A, x)]
    for args in calls:
        said = []
        for way in (plain, lambda *a: False):
            monkeypatch.setattr(sparse, "_mul_plain", way)
            with pytest.raises(Exception) as e:
                gsa.mul_(*args)
            said.append((type(e.value), str(e.value)))
        assert said[0] == said[1]
