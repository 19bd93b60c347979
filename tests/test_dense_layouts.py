"""The buffers and leading dimensions that the host layer hands to the library for dense operands:
every element it would read or write is the operand's own, whatever the view."""
import itertools

import numpy as np
import pytest
import torch


def views(r, c):
    """r x c views of storages with distinct elements, in every layout a torch program holds."""
    v = lambda n: torch.arange(1, n + 1, dtype=torch.float64)
    yield "column-major", v(r * c).view(c, r).t()
    yield "row-major", v(r * c).view(r, c)
    yield "padded columns", v((r + 3) * c).view(c, r + 3).t()[:r]
    yield "padded rows", v((c + 2) * r).view(r, c + 2)[:, :c]
    yield "no unit stride", v(2 * r * 2 * c).view(2 * r, 2 * c)[::2, ::2]
    yield "one column repeated", v(r)[:, None].expand(r, c)
    yield "one row repeated", v(c)[None, :].expand(r, c)
    yield "one value", v(1)[0].expand(r, c)
    if r and c:
        yield "overlapping columns", v(r + c - 1).unfold(0, r, 1).t()
        yield "overlapping rows", v(r + c - 1).unfold(0, c, 1)
        yield "half overlapping columns", v(r + (c - 1) * max(r // 2, 1)).unfold(0, r, max(r // 2, 1)).t()


SIZES = [(1, 1), (1, 5), (5, 1), (4, 3), (3, 4), (8, 2), (0, 3), (3, 0)]


def elements(buf, ld, op, rows, cols):
    """op(B) as the library reads it, from buf's first element on; and the last element it touches."""
    i, c = np.meshgrid(np.arange(rows), np.arange(cols), indexing="ij")
    at = i + c * ld if op == 0 else c + i * ld
    flat = torch.as_strided(buf, (buf.untyped_storage().nbytes() // 8 - buf.storage_offset(),), (1,)).numpy()
    assert at.size == 0 or at.max() < flat.size, "past the operand's storage"
    return flat[at]


@pytest.mark.parametrize("r,c", SIZES)
def test_operand(gsa, r, c):
    import genericsparsearrays_gb300.sparse as sparse
    for name, t in views(r, c):
        for wrap in (lambda x: x, gsa.transpose, gsa.adjoint):
            buf, ld, op, rows, cols = sparse._dense_operand(wrap(t))
            want = t.numpy() if wrap(t) is t else t.numpy().T
            assert (rows, cols) == want.shape
            assert ld >= max(rows if op == 0 else cols, 1), name
            assert np.array_equal(elements(buf, ld, op, rows, cols), want), name


@pytest.mark.parametrize("r,c", SIZES)
def test_output(gsa, r, c):
    import genericsparsearrays_gb300.sparse as sparse
    for name, t in views(r, c):
        distinct = np.unique(t.numpy()).size == t.numel()
        try:
            C2, Cw, ld = sparse._output(t)
        except gsa.ArgumentError:
            assert not distinct, name
            continue
        assert ld >= max(r, 1)
        assert np.array_equal(elements(Cw, ld, 0, r, c), t.numpy()), name
        assert distinct or Cw is not C2, name  # nothing is written where two elements lie


@pytest.mark.parametrize("n", [1, 4])
def test_vectors(gsa, n):
    import genericsparsearrays_gb300.sparse as sparse
    for t in (torch.arange(3.0 * n).double()[::3], torch.ones(1, dtype=torch.float64).expand(n)):
        buf, ld, op, rows, cols = sparse._dense_operand(t)
        assert np.array_equal(elements(buf, ld, op, rows, cols)[:, 0], t.numpy())


@pytest.mark.parametrize("r,c", SIZES)
def test_grouped_operands(gsa, r, c):
    """A batch keeps its operands where they are: a layout that no ld describes is refused."""
    from genericsparsearrays_gb300 import batch
    for name, t in views(r, c):
        described = False
        try:
            k, ld, rowmajor = batch._dense_in(t)
            described = True
        except gsa.ArgumentError:
            pass
        if described:
            assert k == c
            assert np.array_equal(elements(t, ld, rowmajor, r, c), t.numpy()), name
        try:
            k, ld = batch._column_major(t, "C")
        except gsa.ArgumentError:
            continue
        assert k == c and np.array_equal(elements(t, ld, 0, r, c), t.numpy()), name
        assert np.unique(t.numpy()).size == t.numel(), name
    strided = torch.arange(3.0 * r).double()[::3]
    if r > 1:
        assert batch._dense_in(strided) == (1, 3, 1)
        with pytest.raises(gsa.ArgumentError):
            batch._column_major(strided, "C")


@pytest.mark.gpu
@pytest.mark.parametrize("r,c", [(5, 1), (1, 5), (40, 3), (3, 40)])
def test_products(gsa, cuda, r, c):
    """Both ways of mul_, on B of every layout, against a dense product of integers."""
    rng = np.random.default_rng(r)
    m, nnz = 23, 4 * r
    D = np.zeros((m, r))
    rows, cols, vals = rng.integers(0, m, nnz), rng.integers(0, r, nnz), rng.integers(-4, 5, nnz).astype(np.float64)
    np.add.at(D, (rows, cols), vals)
    A = gsa.GenericSparseMatrixCSR(gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(m, r, rows + 1, cols + 1, vals)))
    for name, t in views(r, c):
        B = torch.as_strided(torch.arange(1, 2000, dtype=torch.float64, device=cuda), t.shape, t.stride())
        want = D @ B.cpu().numpy()
        for _ in range(2):  # the second call finds the plan made
            C = torch.empty((c, m), dtype=torch.float64, device=cuda).t()
            assert np.array_equal(gsa.mul_(C, A, B).cpu().numpy(), want), name
    if c > 1:
        for C in (torch.zeros(m, dtype=torch.float64, device=cuda)[:, None].expand(m, c),
                  torch.zeros(m + c - 1, dtype=torch.float64, device=cuda).unfold(0, m, 1).t()):
            with pytest.raises(gsa.ArgumentError):
                gsa.mul_(C, A, torch.zeros((c, r), dtype=torch.float64, device=cuda).t())


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.float64, torch.complex128])
def test_subclass_of_adjoint(gsa, cuda, dt):
    """A wrapper derived from Adjoint is the adjoint in every call, not in the first alone."""
    class Mine(gsa.Adjoint):
        pass
    v = torch.tensor([1 + 2j, 3 - 1j, -2 + 0.5j]).to(dt) if dt.is_complex else torch.tensor([1.0, 3.0, -2.0]).to(dt)
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(2, 3, np.array([1, 3, 4]), np.array([1, 3, 2]), v))
    x = torch.tensor([2.0, -1.0], dtype=dt, device=cuda)
    want = gsa.mul(gsa.adjoint(A), x)
    for _ in range(3):
        y = gsa.mul_(torch.empty(3, dtype=dt, device=cuda), Mine(A), x)
        assert torch.equal(y, want)
