"""Plans made on the GPU: their counts against a numpy restatement of the rules, and the products
that run on them against exact integer sums, at the edges of the passes (32-row warps, 4096-row
CTAs, 32768-row segments) and of the rules (rows of 32, 33, 512, 513 and many thousand entries)."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CHUNK, PLAN_LEN, SEGMENT = 512, 32, 32768


def lanes(length):
    g = 1
    while 32 * g < length:
        g *= 2
    return g


def expected(length):
    """max_len, rows the plan takes, chunks, bin-order warps of a plan of these row lengths."""
    n = length.size
    pad = np.zeros(-(-n // 32) * 32, np.int64)
    pad[:n] = length
    w = pad.reshape(-1, 32)
    nat = (w > CHUNK) | ((w > PLAN_LEN) & (8 * w > w.sum(1, keepdims=True)))
    left = np.where(nat, 0, w)
    total = left.sum(1)
    held = 0
    for row, t in zip(left, total):
        g = 1
        while g < 32 and (t >> 5) > 6 * g:
            g *= 2
        held += 32 * int((-(-row.reshape(g, 32 // g).max(1) // g)).sum())
    binned = n >= 32 and held > 0 and total.sum() / held < 0.9
    rows = pad[nat.ravel()] if not binned else length[length > CHUNK]
    warps = 0
    if binned:
        for s in range(0, n, SEGMENT):
            seg = length[s:s + SEGMENT]
            seg = seg[seg <= CHUNK]
            for g in (1, 2, 4, 8, 16):
                k = sum(1 for x in seg if lanes(x) == g)
                warps += -(-k // (32 // g))
    return int(length.max(initial=0)), n if binned else int(nat.sum()), int((-(-rows // CHUNK)).sum()), warps


def lengths_of(kind, n, rng):
    if kind == "even":
        return np.full(n, 5)
    if kind == "edges":
        return rng.choice([0, 1, 31, 32, 33, 63, 64, 65, 256, 257, 511, 512, 513], n)
    if kind == "one_long":
        x = rng.poisson(4, n)
        x[n // 2] = 40_000 if n > 1000 else 600
        return x
    return np.minimum(np.ceil(3 * rng.uniform(0, 1, n) ** (-1 / 1.5)), 5000)  # power law


@pytest.mark.parametrize("it", [np.int32, np.int64])
@pytest.mark.parametrize("kind", ["even", "edges", "one_long", "power"])
@pytest.mark.parametrize("n", [1, 31, 33, 4095, 4097, 32769, 70_001])
def test_plan_counts_and_products(gsa, cuda, n, kind, it):
    rng = np.random.default_rng(n + len(kind))
    length = lengths_of(kind, n, rng).astype(np.int64)
    inner = 60_000
    rowptr = np.concatenate([[0], np.cumsum(length)])
    nnz = int(rowptr[-1])
    cols = rng.integers(0, inner, nnz)
    vals = rng.integers(-8, 9, nnz).astype(np.float64)
    x = rng.integers(-8, 9, inner).astype(np.float64)
    want = np.add.reduceat(np.append(vals * x[cols], 0.0), np.minimum(rowptr[:-1], nnz)) * (length > 0)
    for dt in (np.float64, np.complex128):  # natural order; bin order where the plan has one
        A = gsa.GenericSparseMatrixCSR(n, inner, (rowptr + 1).astype(it), (cols + 1).astype(it), vals.astype(dt))
        A = gsa.adapt(cuda, A)
        y = (A @ torch.from_numpy(x.astype(dt)).to(cuda)).cpu().numpy()
        assert np.array_equal(y, want.astype(dt))
    max_len, nlong, nchunks, warps = expected(length)
    lib = gsa._lib.load()
    h = ctypes.c_void_p(0)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.gsa_plan_create(stream, gsa._lib.IDX32 if it == np.int32 else gsa._lib.IDX64, n, nnz,
                               ctypes.c_void_p(A.rowptr.data_ptr()), 1, ctypes.byref(h)) == 0
    got = [ctypes.c_int64(-1) for _ in range(3)]
    lib.gsa_plan_info(h, *[ctypes.byref(g) for g in got])
    view, bw = ctypes.c_void_p(0), ctypes.c_int64(-1)
    lib.gsa_plan_bin_order(h, ctypes.byref(view), ctypes.byref(bw))
    lib.gsa_plan_destroy(h)
    assert [g.value for g in got] == [max_len, nlong, nchunks]
    assert bw.value == (warps if max_len <= CHUNK else 0)


@pytest.mark.parametrize("it", [np.int32, np.int64])
@pytest.mark.parametrize("rows,m", [
    ([0, 1, 1, 33, 34, 66, 99, 5000, 5000, 9999], 10_000),  # gaps of 31 to 33 rows and long ones
    ([7], 100_000), ([99_999], 100_000), ([], 77), ([0, 0, 0], 1),
    (list(range(0, 64 * 33, 33)), 64 * 33),                  # a wide gap before every lane of two warps
])
def test_coo_row_pointers_with_gaps(gsa, cuda, rows, m, it):
    n = 50
    r = np.asarray(rows, np.int64)
    c = np.arange(r.size) * 7 % n
    v = (np.arange(r.size) + 1.0)
    x = np.arange(n) - 20.0
    want = np.zeros(m)
    np.add.at(want, r, v * x[c])
    xd = torch.from_numpy(x).to(cuda)
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(m, n, (r + 1).astype(it), (c + 1).astype(it), v))
    assert np.array_equal((A @ xd).cpu().numpy(), want)
    if r.size > 1 and r[0] != r[-1]:  # one decrease, at the end: not sorted
        p = np.concatenate([np.arange(1, r.size), [0]])
        B = gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(m, n, (r[p] + 1).astype(it), (c[p] + 1).astype(it), v[p]))
        assert np.array_equal((B @ xd).cpu().numpy(), want)
        assert B._plan is None
