"""COO -> CSR / CSC and COO sums around the sizes at which a row changes hands (16, 256, one chunk of
4096 entries, several), with repeated positions, against a stable numpy sort."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = {
    "edges": [0, 1, 15, 16, 17, 31, 32, 33, 255, 256, 257, 511, 513, 1024, 1025],
    "chunks": [4095, 4096, 4097, 8191, 8192, 8193, 5, 12289, 300],
    "one_row": [70_001],
}


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex128])
@pytest.mark.parametrize("it", [np.int32, np.int64])
@pytest.mark.parametrize("kind", sorted(LENGTHS))
@pytest.mark.parametrize("filler", [0, 40_000])  # rows of about 12 entries around them: many buckets
def test_conversion_of_long_rows(gsa, cuda, kind, filler, it, dt):
    rng = np.random.default_rng(len(kind) + filler)
    lens = np.concatenate([rng.poisson(12, filler // 2), LENGTHS[kind], rng.poisson(12, filler - filler // 2)])
    m, n = lens.size, 3000
    rows = np.repeat(np.arange(m), lens)
    cols = rng.integers(0, n, rows.size)  # repeats inside rows: their input order is kept
    p = rng.permutation(rows.size)
    rows, cols = rows[p], cols[p]
    vals = np.arange(rows.size).astype(dt)
    order = np.lexsort((cols, rows))
    for cls, a, b in ((gsa.GenericSparseMatrixCSR, rows, cols), (gsa.GenericSparseMatrixCSC, cols, rows)):
        shape = (m, n) if cls is gsa.GenericSparseMatrixCSR else (n, m)
        A = gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(*shape, (a + 1).astype(it), (b + 1).astype(it), vals)
                      if cls is gsa.GenericSparseMatrixCSR else
                      gsa.GenericSparseMatrixCOO(*shape, (cols + 1).astype(it), (rows + 1).astype(it), vals))
        M = cls(A)
        ptr, idx = (M.rowptr, M.colval) if cls is gsa.GenericSparseMatrixCSR else (M.colptr, M.rowval)
        assert np.array_equal(ptr.cpu().numpy(), np.concatenate([[0], np.cumsum(lens)]) + 1)
        assert np.array_equal(idx.cpu().numpy(), cols[order] + 1)
        assert np.array_equal(M.nzval.cpu().numpy(), vals[order])


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128, np.int64])
@pytest.mark.parametrize("kind", sorted(LENGTHS))
def test_sum_of_long_columns(gsa, cuda, kind, dt):
    """A + transpose(A) + lambda * I of integer values: exact sums, zeros dropped, column-major."""
    rng = np.random.default_rng(len(kind))
    lens = np.asarray(LENGTHS[kind])
    n = 3001
    cols = np.repeat(rng.integers(0, n, lens.size), lens)
    rows = rng.integers(0, n, cols.size)
    p = rng.permutation(cols.size)
    rows, cols = rows[p], cols[p]
    vals = rng.integers(-3, 4, rows.size)
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(n, n, rows + 1, cols + 1, vals.astype(dt)))
    C = (A + gsa.transpose(A)) + gsa.UniformScaling(2)
    dense = np.zeros((n, n), np.int64)
    np.add.at(dense, (rows, cols), vals)
    dense = dense + dense.T
    # A + transpose(A) drops its zeros; adding 2 I drops the diagonal's
    dense[np.arange(n), np.arange(n)] += 2
    c, r = np.nonzero(dense.T)
    assert np.array_equal(C.rowind.cpu().numpy(), r + 1) and np.array_equal(C.colind.cpu().numpy(), c + 1)
    assert np.array_equal(C.nzval.cpu().numpy(), dense[r, c].astype(dt))
