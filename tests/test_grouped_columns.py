"""Columns per thread of a batch that leaves them open: chosen by its items for ComplexF64, by the type
otherwise; and the products at the chosen width."""
import ctypes

import numpy as np
import pytest
import torch


def columns(gsa, dtype, items):
    """gsa_grouped_columns of (columns, entries, row-major) items."""
    from genericsparsearrays_gb300 import batch
    a = np.zeros(len(items), batch.ITEM_DTYPE)
    for row, (k, nnz, rowmajor) in zip(a, items):
        row["k"], row["nnz"], row["b_rowmajor"], row["m"], row["n"] = k, nnz, rowmajor, 100, 100
    return gsa._lib.load().gsa_grouped_columns(dtype, a.ctypes.data_as(ctypes.c_void_p), a.size)


@pytest.mark.parametrize("rowmajor", [0, 1])
def test_complex64_by_its_items(gsa, rowmajor):
    L = gsa._lib
    for k, want in ((1, 1), (2, 1), (3, 1), (4, 2), (8, 2), (16, 2)):
        assert columns(gsa, L.C64, [(k, 1000, rowmajor)] * 5) == want
    assert columns(gsa, L.C64, [(k, 900, rowmajor) for k in (1, 4, 8)]) == (2 if rowmajor else 1)
    assert columns(gsa, L.C64, [(1, 10**6, rowmajor), (8, 10, rowmajor)]) == 1  # the work decides
    assert columns(gsa, L.C64, [(1, 10, rowmajor), (8, 10**6, rowmajor)]) == 2


def test_other_types_by_type(gsa):
    L = gsa._lib
    for dtype, want in ((L.F32, 4), (L.I32, 4), (L.F64, 2), (L.C32, 2), (L.I64, 2)):
        assert columns(gsa, dtype, [(8, 1000, 1)]) == want
    assert columns(gsa, L.C64, []) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["column-major", "row-major"])
@pytest.mark.parametrize("ks", [(1,), (3,), (8,), (1, 4, 8), (1, 5, 16)])
def test_products_at_the_chosen_width(gsa, cuda, ks, layout):
    from genericsparsearrays_gb300 import batch
    rng = np.random.default_rng(len(ks))
    products, wants = [], []
    for i in range(12):
        n, k = int(rng.integers(1, 400)), ks[i % len(ks)]
        nnz = 6 * n
        r, c = np.sort(rng.integers(0, n, nnz)), rng.integers(0, n, nnz)
        v = rng.integers(-4, 5, nnz) + 1j * rng.integers(-4, 5, nnz)
        ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]) + 1
        A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(n, n, ptr.astype(np.int64), (c + 1).astype(np.int64), v))
        X = rng.integers(-4, 5, (n, k)) + 1j * rng.integers(-4, 5, (n, k))
        D = np.zeros((n, n), complex)
        np.add.at(D, (r, c), v)
        B = torch.from_numpy(X).to(cuda)
        B = B if layout == "row-major" else B.t().contiguous().t()
        products.append((A, B, torch.full((k, n), 9, dtype=torch.complex128, device=cuda).t(), 1, 0))
        wants.append(D @ X)
    b = batch.BatchedMul(products)
    launcher = batch.GroupedLauncher(cuda)
    for run in (lambda: b.run("grouped"), lambda: b.run("graph"), lambda: b.run("per_call"),
                lambda: launcher.launch(products)):
        for _, _, C, _, _ in products:
            C.fill_(9)
        run()
        torch.cuda.synchronize()
        for (_, _, C, _, _), want in zip(products, wants):
            assert np.array_equal(C.cpu().numpy(), want)
