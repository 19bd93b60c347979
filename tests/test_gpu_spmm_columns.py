"""SpMM with every split of the columns into launches and groups: column counts around the widths
(1, 2, 4, 8, 16), both layouts of B, short rows (a lane each), longer ones and chunked ones, against
exact integer sums; and a matrix without columns."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

KS = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 33]


@pytest.mark.parametrize("rows", ["short", "longer", "chunked"])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128, np.int32, np.int64])
def test_every_column_split(gsa, cuda, dt, rows):
    rng = np.random.default_rng(len(rows))
    m, n = 700, 900
    lens = {"short": rng.integers(0, 7, m), "longer": rng.integers(0, 40, m), "chunked": rng.integers(0, 12, m)}[rows]
    if rows == "chunked":
        lens[[3, 600]] = [1400, 40]
    ptr = np.concatenate([[0], np.cumsum(lens)])
    cols = rng.integers(0, n, ptr[-1])
    vals = rng.integers(-4, 5, ptr[-1]).astype(dt)
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(m, n, (ptr + 1).astype(np.int32), (cols + 1).astype(np.int32), vals))
    dense = np.zeros((m, n), np.float64)
    np.add.at(dense, (np.repeat(np.arange(m), lens), cols), vals.real.astype(np.float64))
    X = rng.integers(-4, 5, (n, max(KS))).astype(dt)
    want = dense @ X.real.astype(np.float64)  # |sums| < 2^24: exact in every type
    for k in KS:
        Xr = torch.from_numpy(X[:, :k].copy()).to(cuda)
        for B in (Xr.t().contiguous().t(), Xr):  # column-major, row-major
            Y = torch.full((k, m), 7, dtype=Xr.dtype, device=cuda).t()
            gsa.mul_(Y, A, B, 2, 3)
            assert np.array_equal(Y.cpu().numpy(), (2 * want[:, :k] + 21).astype(dt)), k


@pytest.mark.parametrize("k", [1, 2, 5, 16])
def test_no_columns(gsa, cuda, k):
    """n = 0 with stored entries (all outside): nothing is read of B, beta*C is what is left."""
    for dt in (np.float32, np.float64, np.complex128):
        A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(3, 0, np.array([1, 2, 2, 4]), np.array([1, 1, 2]),
                                                       np.ones(3, dt)))
        C = torch.ones((k, 3), dtype=torch.from_numpy(np.zeros(1, dt)).dtype, device=cuda).t()
        gsa.mul_(C, A, torch.empty((k, 0), dtype=C.dtype, device=cuda).t(), 1, 2)
        assert np.array_equal(C.cpu().numpy(), np.full((3, k), 2, dt))


@pytest.mark.parametrize("fmt", ["csr", "csc", "coo"])
@pytest.mark.parametrize("k", [1, 3])
def test_complex_alpha_one_keeps_special_values(gsa, cuda, fmt, k):
    """alpha = 1 + 0i is not multiplied where that changes no bit; infinities, NaN and -0 come out as
    the product with alpha gives them: as alpha = 2 + 0i gives them, halved."""
    s = np.array([0.0, -0.0, 1.5, -2.25, np.inf, -np.inf, np.nan])
    x = np.empty((7, 7), np.complex128)
    x.real, x.imag = np.meshgrid(s, s)
    x = np.repeat(x.reshape(-1, 1), k, 1)
    n = x.shape[0]
    p = np.random.default_rng(0).permutation(n) if fmt == "coo" else np.arange(n)
    eye = np.arange(1, n + 1)
    cls = {"csr": gsa.GenericSparseMatrixCSR, "csc": gsa.GenericSparseMatrixCSC, "coo": gsa.GenericSparseMatrixCOO}[fmt]
    ptr = eye[p] if fmt == "coo" else np.arange(1, n + 2)
    A = gsa.adapt(cuda, cls(n, n, ptr, eye[p], np.ones(n, np.complex128)))
    X = torch.from_numpy(np.asfortranarray(x)).to(cuda)
    one, two = (gsa.mul_(torch.zeros_like(X), A, X, al, 0).cpu().numpy().copy().view(np.float64) for al in (1, 2))
    assert np.array_equal(one, two / 2, equal_nan=True)
    assert np.array_equal(np.signbit(one) & ~np.isnan(one), np.signbit(two) & ~np.isnan(two))
