"""SpGEMM rows around the sizes at which they change kernels (8 entries; 16 written together; 32 and
256 products), sorted and unsorted Q rows, repeated columns, against exact integer products."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("it", [np.int32, np.int64])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128, np.int32, np.int64])
@pytest.mark.parametrize("order", ["sorted", "unsorted", "repeats"])
@pytest.mark.parametrize("fmt", ["csr", "csc"])
def test_row_classes(gsa, cuda, fmt, order, dt, it):
    rng = np.random.default_rng(len(order))
    k, n = 130, 5000
    qlen = np.concatenate([[0, 1, 2, 3, 4, 5, 8, 15, 16, 17, 31, 32, 33, 40, 200], rng.integers(0, 7, k - 15)])
    qptr = np.concatenate([[0], np.cumsum(qlen)])
    rows = []
    for l in qlen:
        c = rng.choice(n, l, replace=False) if order != "repeats" else rng.integers(0, 12, l)
        rows.append(np.sort(c) if order != "unsorted" else c)
    qcol = np.concatenate(rows).astype(np.int64)
    plen = np.concatenate([[0, 1, 1, 2, 7, 8, 9, 40], rng.integers(0, 11, 300)])
    pcol = [np.sort(rng.choice(k, min(l, k), replace=False)) for l in plen]
    for r, q in ((1, [7]), (2, [10])):  # one entry selecting a row of 15 and of 31 products
        pcol[r] = np.array(q)
    pcol.append(np.arange(5, 9))
    plen = np.array([c.size for c in pcol])
    m = plen.size
    pptr = np.concatenate([[0], np.cumsum(plen)])
    pidx = np.concatenate(pcol).astype(np.int64)
    pv, qv = rng.integers(1, 5, pidx.size), rng.integers(-3, 4, qcol.size)  # zero sums are stored

    def dense(ptr, idx, val, shape):
        D = np.zeros(shape, np.int64)
        np.add.at(D, (np.repeat(np.arange(shape[0]), np.diff(ptr)), idx), val)
        return D
    want = dense(pptr, pidx, pv, (m, k)) @ dense(qptr, qcol, qv, (k, n))
    reach = (dense(pptr, pidx, np.ones_like(pv), (m, k)) @ dense(qptr, qcol, np.ones_like(qv), (k, n))) > 0
    t = lambda a: (a + 1).astype(it)
    if fmt == "csr":
        P = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(m, k, t(pptr), t(pidx), pv.astype(dt)))
        Q = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(k, n, t(qptr), t(qcol), qv.astype(dt)))
        C = P @ Q
        ptr, idx = C.rowptr, C.colval
    else:  # the transposed product: columns of the second factor select columns of the first
        P = gsa.adapt(cuda, gsa.GenericSparseMatrixCSC(k, m, t(pptr), t(pidx), pv.astype(dt)))
        Q = gsa.adapt(cuda, gsa.GenericSparseMatrixCSC(n, k, t(qptr), t(qcol), qv.astype(dt)))
        C = Q @ P
        ptr, idx = C.colptr, C.rowval
    r, c = np.nonzero(reach)
    assert np.array_equal(ptr.cpu().numpy(), np.concatenate([[0], np.cumsum(reach.sum(1))]) + 1)
    assert np.array_equal(idx.cpu().numpy(), c + 1)
    assert np.array_equal(C.nzval.cpu().numpy(), want[r, c].astype(dt))
