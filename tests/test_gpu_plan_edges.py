"""Plans at the sizes where their passes change form: one CTA up to 8192 rows, whose sums go straight
to host memory; CTAs of 2048 rows with cleared totals beyond; segments of 32768 rows."""
import ctypes

import numpy as np
import pytest
import torch

from test_gpu_plan import CHUNK, expected, lengths_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["edges", "one_long", "power"])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 8191, 8192, 8193, 10239, 10240, 10241, 32767, 32768])
def test_sizes_of_the_passes(gsa, cuda, n, kind):
    rng = np.random.default_rng(n)
    length = lengths_of(kind, n, rng).astype(np.int64)
    inner = 50_000
    rowptr = np.concatenate([[0], np.cumsum(length)])
    nnz = int(rowptr[-1])
    cols, vals = rng.integers(0, inner, nnz), rng.integers(-8, 9, nnz).astype(np.float64)
    x = rng.integers(-8, 9, inner).astype(np.float64)
    want = np.add.reduceat(np.append(vals * x[cols], 0.0), np.minimum(rowptr[:-1], nnz)) * (length > 0)
    lib = gsa._lib.load()
    for dt in (np.float64, np.complex128):
        A = gsa.GenericSparseMatrixCSR(n, inner, (rowptr + 1).astype(np.int32), (cols + 1).astype(np.int32), vals.astype(dt))
        A = gsa.adapt(cuda, A)
        y = (A @ torch.from_numpy(x.astype(dt)).to(cuda)).cpu().numpy()
        assert np.array_equal(y, want.astype(dt))
    max_len, nlong, nchunks, warps = expected(length)
    for _ in range(2):  # the second plan's counts go where the first one's lie
        h, got = ctypes.c_void_p(0), [ctypes.c_int64(-1) for _ in range(3)]
        assert lib.gsa_plan_create(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), gsa._lib.IDX32, n, nnz,
                                   ctypes.c_void_p(A.rowptr.data_ptr()), 1, ctypes.byref(h)) == 0
        lib.gsa_plan_info(h, *[ctypes.byref(g) for g in got])
        view, bw = ctypes.c_void_p(0), ctypes.c_int64(-1)
        lib.gsa_plan_bin_order(h, ctypes.byref(view), ctypes.byref(bw))
        lib.gsa_plan_destroy(h)
        assert [g.value for g in got] == [max_len, nlong, nchunks]
        assert bw.value == (warps if max_len <= CHUNK else 0)


@pytest.mark.parametrize("dt", [np.float64, np.complex64, np.int64])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 15, 16, 17, 24, 25, 32])
def test_merged_rows_of_every_length(gsa, cuda, count, dt):
    """SpGEMM rows whose results have exactly `count` entries, beside rows of none and of 32: eight
    are written together."""
    n, m = 40, 100
    rng = np.random.default_rng(count)
    qlen = np.zeros(n, np.int64)
    qlen[:4], qlen[4:8] = count // 4, 8
    qlen[:count % 4] += 1
    qptr = np.concatenate([[0], np.cumsum(qlen)])
    qcol = np.concatenate([np.arange(l) * 8 + i % 8 for i, l in enumerate(qlen)])  # the rows interleave, none meet
    width = 80
    rows = [[0, 1, 2, 3] if i % 3 == 0 else ([] if i % 3 == 1 else [4, 5, 6, 7]) for i in range(m)]
    pptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    pidx = np.concatenate([np.array(r, np.int64) for r in rows])
    pv, qv = rng.integers(1, 9, pidx.size), rng.integers(1, 9, qcol.size)
    P = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(m, n, (pptr + 1).astype(np.int32), (pidx + 1).astype(np.int32), pv.astype(dt)))
    Q = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(n, width, (qptr + 1).astype(np.int32), (qcol + 1).astype(np.int32), qv.astype(dt)))
    D, E = np.zeros((m, n), np.int64), np.zeros((n, width), np.int64)
    D[np.repeat(np.arange(m), np.diff(pptr)), pidx] = pv
    E[np.repeat(np.arange(n), qlen), qcol] = qv
    want = D @ E
    r, c = np.nonzero(want)
    C = P @ Q
    assert np.array_equal(np.diff(C.rowptr.cpu().numpy())[::3], np.full((m + 2) // 3, count))
    assert np.array_equal(C.colval.cpu().numpy(), c + 1)
    assert np.array_equal(C.nzval.cpu().numpy(), want[r, c].astype(dt))
