"""Buckets too large for the shared staging, among rows of one entry: their rows of every length up to
20 sorted in global memory, against numpy's stable sort."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex128])
@pytest.mark.parametrize("it", [np.int32, np.int64])
@pytest.mark.parametrize("longest", [8, 16, 20])
def test_rows_of_an_oversized_bucket(gsa, cuda, longest, it, dt):
    rng = np.random.default_rng(longest)
    n = 200_000
    length = np.ones(n, np.int64)
    length[1000:4000] = rng.integers(longest - 7, longest + 1, 3000)  # some 36,000 entries in two buckets
    r = np.repeat(np.arange(n), length)
    c = rng.integers(0, n, r.size)
    c[::7] = c[0]  # repeated positions keep their order
    p = rng.permutation(r.size)
    r, c, v = r[p], c[p], rng.integers(1, 9, r.size).astype(dt)
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(n, n, (r + 1).astype(it), (c + 1).astype(it), v))
    X = gsa.GenericSparseMatrixCSR(A)
    order = np.lexsort((c, r))
    assert np.array_equal(X.rowptr.cpu().numpy(), np.concatenate([[0], np.cumsum(length)]) + 1)
    assert np.array_equal(X.colval.cpu().numpy(), c[order] + 1)
    assert np.array_equal(X.nzval.cpu().numpy(), v[order])
    S = gsa.transpose(A) + gsa.transpose(A)  # the sort without values: columns of the sum are A's rows
    key, inv = np.unique(r * n + c, return_inverse=True)
    want = np.bincount(inv, weights=2 * v.real)
    assert np.array_equal(S.colind.cpu().numpy(), key // n + 1)
    assert np.array_equal(S.rowind.cpu().numpy(), key % n + 1)
    assert np.array_equal(S.nzval.cpu().numpy(), want.astype(dt))
