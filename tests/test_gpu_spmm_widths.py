"""SpMM at an explicit width (GSA_TUNE_SPMM_COLUMNS) and at the library's own, for column counts that
no width divides, against exact integer sums; a B too wide for L2 by its layout alone."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def width(gsa):
    lib = gsa._lib.load()
    yield lambda w: lib.gsa_set_tuning(gsa._lib.TUNE_SPMM_COLUMNS, w)
    lib.gsa_set_tuning(gsa._lib.TUNE_SPMM_COLUMNS, 0)


@pytest.mark.parametrize("rows", ["grid", "forty", "uneven"])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128, np.int32, np.int64])
def test_widths(gsa, cuda, width, dt, rows):
    rng = np.random.default_rng(len(rows))
    m, n = 300, 500
    lens = {"grid": np.full(m, 5), "forty": np.full(m, 40), "uneven": rng.integers(0, 40, m)}[rows]
    lens[7] = 1100 if rows == "uneven" else lens[7]
    ptr = np.concatenate([[0], np.cumsum(lens)])
    cols, vals = rng.integers(0, n, ptr[-1]), rng.integers(-4, 5, ptr[-1]).astype(dt)
    D = np.zeros((m, n))
    np.add.at(D, (np.repeat(np.arange(m), lens), cols), vals.real.astype(np.float64))
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(m, n, (ptr + 1).astype(np.int32), (cols + 1).astype(np.int32), vals))
    for k in (2, 3, 5, 6, 7, 9, 10, 11, 12, 13, 14, 15, 18, 21, 23, 24, 25, 29, 31, 35):
        X = rng.integers(-4, 5, (n, k)).astype(dt)
        want = (D @ X.real.astype(np.float64)).astype(dt)
        wantT = (D.T @ X[:m].real.astype(np.float64)).astype(dt)
        Xr = torch.from_numpy(X).to(cuda)
        for w in (0, 1, 2, 4, 8):
            assert width(w) == 0
            for B in (Xr.t().contiguous().t(), Xr):
                Y = torch.full((k, m), 7, dtype=Xr.dtype, device=cuda).t()
                assert np.array_equal(gsa.mul_(Y, A, B).cpu().numpy(), want), (k, w)
            Z = torch.full((k, n), 7, dtype=Xr.dtype, device=cuda).t()
            assert np.array_equal(gsa.mul_(Z, gsa.transpose(A), Xr[:m].t().contiguous().t()).cpu().numpy(), wantT), (k, w)


@pytest.mark.parametrize("dt", [torch.float64, torch.int64])
@pytest.mark.parametrize("k", [3, 7, 8, 9])
def test_wide_operand(gsa, cuda, dt, k):
    """More bytes of B than stay in L2: pairs of columns, an odd one at the end."""
    n, per = 2_100_000, 8
    g = torch.Generator(device=cuda).manual_seed(k)
    cols = torch.randint(0, n, (n * per,), generator=g, device=cuda)
    vals = torch.randint(-3, 4, (n * per,), generator=g, device=cuda).to(dt)
    A = gsa.GenericSparseMatrixCSR(n, n, torch.arange(0, n * per + 1, per, device=cuda) + 1, cols + 1, vals)
    X = torch.randint(-3, 4, (k, n), generator=g, device=cuda).to(dt).t()
    Y = gsa.mul_(torch.empty((k, n), dtype=dt, device=cuda).t(), A, X)
    for c in range(k):
        want = (vals * X[:, c][cols]).view(n, per).sum(1)
        assert torch.equal(Y[:, c], want)
