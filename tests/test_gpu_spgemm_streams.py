"""A SpGEMM handle whose calls come on several streams, or under capture, and that is destroyed at
once: its memory stays with the work that reads it."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


class Product:
    """A * A in CSR with rows of every kind (merged, listed, small, big), and its handle."""

    def __init__(self, gsa, cuda, n=3000):
        rng = np.random.default_rng(n)
        length = rng.integers(0, 8, n)
        length[:4] = [12, 40, 90, 200]
        rowptr = np.concatenate([[0], np.cumsum(length)])
        cols = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in length])
        self.A = A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(
            n, n, (rowptr + 1).astype(np.int32), (cols + 1).astype(np.int32), rng.standard_normal(cols.size)))
        self.want = A @ A
        self.lib, self.gsa, self.cuda = gsa._lib.load(), gsa, cuda
        torch.cuda.synchronize()

    def create(self, stream):
        A, g = self.A, self.gsa._lib
        self.ptr_c = torch.zeros(A.m + 1, dtype=torch.int32, device=self.cuda)
        torch.cuda.synchronize()
        nnz, self.handle = ctypes.c_int64(0), ctypes.c_void_p(0)
        arrays = (ptr(A.rowptr), ptr(A.colval), ptr(A.nzval), A.nzval.numel())
        assert self.lib.gsa_spgemm_create(ctypes.c_void_p(stream.cuda_stream), 0, g.F64, g.IDX32, A.m, A.n, A.n,
                                          *arrays, *arrays, 1, ptr(self.ptr_c), ctypes.byref(nnz),
                                          ctypes.byref(self.handle)) == 0
        assert nnz.value == self.want.nzval.numel()

    def outputs(self):
        nnz = self.want.nzval.numel()
        return (torch.zeros(nnz, dtype=torch.int32, device=self.cuda),
                torch.zeros(nnz, dtype=torch.float64, device=self.cuda))

    def compute(self, stream, out):
        assert self.lib.gsa_spgemm_compute(ctypes.c_void_p(stream.cuda_stream), self.handle, ptr(out[0]),
                                           ptr(out[1])) == 0

    def destroy(self):
        assert self.lib.gsa_spgemm_destroy(self.handle) == 0

    def check(self, out):
        assert torch.equal(self.ptr_c, self.want.rowptr)
        assert torch.equal(out[0], self.want.colval) and torch.equal(out[1], self.want.nzval)


@pytest.mark.parametrize("late", ["create", "first", "second", "none"])
def test_streams_ordered_by_the_api_alone(gsa, cuda, late):
    p = Product(gsa, cuda)
    streams = {name: torch.cuda.Stream() for name in ("create", "first", "second")}
    p.create(streams["create"])
    outs = p.outputs(), p.outputs()
    torch.cuda.synchronize()
    if late != "none":  # about 50 ms of waiting before that stream's part
        with torch.cuda.stream(streams[late]):
            torch.cuda._sleep(100_000_000)
    p.compute(streams["first"], outs[0])
    p.compute(streams["second"], outs[1])
    p.destroy()
    spare = [Product(gsa, cuda, n) for n in (2000, 3000, 4000)]  # take what the pool has been given
    torch.cuda.synchronize()
    for out in outs:
        p.check(out)
    assert all(q.want.nzval.numel() for q in spare)


def test_captured_compute(gsa, cuda):
    """The graph's replays read the handle's memory until it is destroyed."""
    p = Product(gsa, cuda)
    p.create(torch.cuda.current_stream())
    out = p.outputs()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.compute(torch.cuda.current_stream(), out)
    for _ in range(2):
        for t in out:
            t.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(20_000_000)
            graph.replay()
    p.destroy()  # waits for the replay
    p.check(out)
