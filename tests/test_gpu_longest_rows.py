"""Rows of so many entries that their chunks are merged in groups, in one further pass or in two,
against torch's stable sort; beside long rows that the first pass finishes, and short ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,nnz", [
    (1, (1 << 24) + 1),        # one row, just beyond the single pass: 65 groups of 64 chunks
    (1, 1 << 24),              # the single pass at its longest
    (3, 20_000_003),           # rows of some 6.7M entries
    (90, 20_000_003),          # about 54 chunks each: one group
    (4, (1 << 26) + 12_345),   # two further passes launched, the second with nothing left
    (1, (1 << 26) + 4097),     # two runs for the second further pass
])
@pytest.mark.parametrize("dt", [torch.int32, torch.complex128])
def test_rows_of_many_chunks(gsa, cuda, rows, nnz, dt):
    if dt.is_complex and nnz > 1 << 25:
        pytest.skip("the same kernels, 10 GB")
    g = torch.Generator(device=cuda).manual_seed(nnz)
    m, n = rows + 1000, 1 << 30
    r = torch.randint(0, rows, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    few = 50_000  # of them in short rows
    r[torch.randint(0, nnz, (few,), generator=g, device=cuda)] = torch.randint(
        0, m, (few,), generator=g, device=cuda, dtype=torch.int32)
    c = torch.randint(0, n, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    v = torch.arange(nnz, dtype=torch.int32, device=cuda).to(dt)
    A = gsa.GenericSparseMatrixCOO(m, n, r + 1, c + 1, v)
    key = r.long() * n + c
    del r, c
    X = gsa.GenericSparseMatrixCSR(A)
    del A
    key, order = torch.sort(key, stable=True)
    assert torch.equal(X.nzval, v[order])
    del order, v
    assert torch.equal(X.colval, (key % n + 1).int())
    rows_at = torch.searchsorted(key, torch.arange(m + 1, device=cuda) * n)
    assert torch.equal(X.rowptr, (rows_at + 1).int())


@pytest.mark.parametrize("nnz", [(1 << 24) + 5, 1 << 20])
def test_sum_of_one_long_column(gsa, cuda, nnz):
    """The sort without values, and the one-level form's buffers: column sums of a long column."""
    g = torch.Generator(device=cuda).manual_seed(nnz)
    m = 1 << 30
    r = torch.randint(0, m, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    c = torch.zeros_like(r)
    v = torch.randint(1, 5, (nnz,), generator=g, device=cuda, dtype=torch.int64)
    A = gsa.GenericSparseMatrixCOO(m, 2, r + 1, c + 1, v)
    Z = gsa.GenericSparseMatrixCOO(m, 2, r[:1] + 1, c[:1] + 2, v[:1])
    S = A + Z
    keys, inv = torch.unique(r, return_inverse=True)
    want = torch.zeros(keys.numel(), dtype=torch.int64, device=cuda).index_add_(0, inv, v)
    assert torch.equal(S.rowind[:-1], keys + 1) and torch.equal(S.nzval[:-1], want)
    assert S.colind[-1].item() == 2 and S.nzval[-1].item() == v[0].item()


def test_one_level_form(gsa, cuda):
    """More rows than the coarse buckets cover, one of them of many chunks."""
    nnz, m = (1 << 24) + 77, 8191 * 4096 + 9
    g = torch.Generator(device=cuda).manual_seed(1)
    r = torch.full((nnz,), m - 3, dtype=torch.int32, device=cuda)
    r[::1000] = torch.randint(0, m, (r[::1000].numel(),), generator=g, device=cuda, dtype=torch.int32)
    c = torch.randint(0, 1 << 30, (nnz,), generator=g, device=cuda, dtype=torch.int32)
    v = torch.arange(nnz, dtype=torch.int32, device=cuda)
    X = gsa.GenericSparseMatrixCSR(gsa.GenericSparseMatrixCOO(m, 1 << 30, r + 1, c + 1, v))
    key, order = torch.sort(r.long() * (1 << 30) + c, stable=True)
    assert torch.equal(X.nzval, v[order])
    assert torch.equal(X.colval, (key % (1 << 30) + 1).int())
