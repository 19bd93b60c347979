"""Plans and SpGEMM handles that are dropped while a stream is being captured by a thread that does
not mind (a thread-local capture of another thread, a relaxed one): the capture goes on, and memory
is given back only after the work that reads it."""
import ctypes
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def matrix(gsa, cuda, n, long, seed=0):
    rng = np.random.default_rng(seed)
    length = rng.integers(0, 6, n)
    length[5] = long
    ptr = np.concatenate([[0], np.cumsum(length)]) + 1
    cols = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in length]) + 1
    A = gsa.adapt(cuda, gsa.GenericSparseMatrixCSR(n, n, ptr.astype(np.int32), cols.astype(np.int32),
                                                   rng.standard_normal(cols.size)))
    x = torch.ones(n, dtype=torch.float64, device=cuda)
    return A, x, gsa.mul(A, x)  # the plan is made


def handle(gsa, cuda, A):
    """An SpGEMM handle with work on two streams."""
    L, lib = gsa._lib, gsa._lib.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    ptr_c, nnz, h = torch.zeros(A.m + 1, dtype=torch.int32, device=cuda), ctypes.c_int64(0), ctypes.c_void_p(0)
    arrays = (p(A.rowptr), p(A.colval), p(A.nzval), A.nzval.numel())
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    assert lib.gsa_spgemm_create(ctypes.c_void_p(streams[0].cuda_stream), 0, L.F64, L.IDX32, A.m, A.n, A.n, *arrays,
                                 *arrays, 1, p(ptr_c), ctypes.byref(nnz), ctypes.byref(h)) == 0
    out = torch.zeros(nnz.value, dtype=torch.int32, device=cuda), torch.zeros(nnz.value, dtype=torch.float64, device=cuda)
    torch.cuda.synchronize()
    assert lib.gsa_spgemm_compute(ctypes.c_void_p(streams[1].cuda_stream), h, p(out[0]), p(out[1])) == 0
    torch.cuda.synchronize()
    return h


@pytest.mark.parametrize("what", ["plan", "coo plan", "spgemm"])
@pytest.mark.parametrize("mode,other", [("thread_local", True), ("relaxed", True), ("relaxed", False)])
def test_dropped_during_a_capture(gsa, cuda, what, mode, other):
    A, x, want = matrix(gsa, cuda, 3000, 700)
    M, _, _ = matrix(gsa, cuda, 3000, 700, 1)
    lib = gsa._lib.load()
    if what == "spgemm":
        h = handle(gsa, cuda, M)
        drop = lambda: lib.gsa_spgemm_destroy(h)
    else:
        if what == "coo plan":
            M = gsa.GenericSparseMatrixCOO(M)
            gsa.mul(M, x)
        plan = M._plan
        h, plan.handle = plan.handle, None
        drop = lambda: lib.gsa_plan_destroy(ctypes.c_void_p(h))
    y, said = torch.zeros_like(x), []
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        gsa.mul_(y, A, x)
        if other:
            t = threading.Thread(target=lambda: said.append(drop()))
            t.start()
            t.join()
        else:
            said.append(drop())
    assert said == [0]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_planning_thread_ends_during_a_capture(gsa, cuda):
    A, x, want = matrix(gsa, cuda, 3000, 700)
    go, planned = threading.Event(), threading.Event()
    kept = []

    def work():
        kept.append(matrix(gsa, cuda, 300, 40))
        torch.cuda.synchronize()
        planned.set()
        go.wait()
    t = threading.Thread(target=work)
    t.start()
    planned.wait()
    y = torch.zeros_like(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        gsa.mul_(y, A, x)
        go.set()
        t.join()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


@pytest.mark.parametrize("what", ["plan", "spgemm"])
def test_dropping_waits_for_every_stream(gsa, cuda, what):
    """No event tells what reads a plan or a handle of several streams: all work has finished."""
    M, x, _ = matrix(gsa, cuda, 3000, 700)
    if what == "spgemm":
        h = handle(gsa, cuda, M)
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # some 50 ms
        done.record()
    assert not done.query()
    if what == "spgemm":
        assert gsa._lib.load().gsa_spgemm_destroy(h) == 0
    else:
        M.__dict__.pop("_plan")
    assert done.query()


def test_threads_that_plan_at_once(gsa, cuda):
    """Small plans of many threads, each with its counts to itself."""
    wrong = []

    def work(seed):
        rng = np.random.default_rng(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            for n, long in ((200, 40), (2000, 600), (300, 290)):
                for _ in range(10):
                    A, x, y = matrix(gsa, cuda, n, long, int(rng.integers(1 << 30)))
                    torch.cuda.current_stream().synchronize()
                    if A._plan is None or A._plan.max_len != long:
                        wrong.append((seed, n))
    threads = [threading.Thread(target=work, args=(s,)) for s in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
