"""Host threads that convert matrices of different sizes at once: no call refuses another's launch.
Buckets of 5000 entries take 100 KB of shared memory, those of the small matrices less than 48 KB."""
import ctypes
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(100, 500_000), (1500, 20_000), (100, 500_000), (1500, 20_000), (2000, 30_000), (60, 300_000), (3000, 60_000),
         (1500, 20_000)]


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
def test_conversions_at_once(gsa, cuda, dt):
    L, lib = gsa._lib, gsa._lib.load()
    code = L.F64 if dt == np.float64 else L.C64
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    calls, checks, kept = [], [], []
    for seed, (n, nnz) in enumerate(SIZES):
        rng = np.random.default_rng(seed)
        r, c, v = rng.integers(0, n, nnz), rng.integers(0, n, nnz), rng.integers(1, 99, nnz).astype(dt)
        rd, cd, vd = (torch.from_numpy(a).to(cuda) for a in ((r + 1).astype(np.int32), (c + 1).astype(np.int32), v))
        po = torch.zeros(n + 1, dtype=torch.int32, device=cuda)
        io, vo = torch.zeros_like(cd), torch.zeros_like(vd)
        size = lib.gsa_coo_to_compressed_workspace_size(0, code, L.IDX32, n, n, nnz)
        ws, stream = torch.empty(size, dtype=torch.uint8, device=cuda), torch.cuda.Stream()
        calls.append((stream, (ctypes.c_void_p(stream.cuda_stream), code, L.IDX32, n, n, nnz, p(rd), p(cd), p(vd), 1,
                               p(po), p(io), p(vo), p(ws), size)))
        order = np.lexsort((c, r))
        checks.append((io, (c[order] + 1).astype(np.int32), vo, v[order]))
        kept.append((rd, cd, vd, po, ws))
    torch.cuda.synchronize()
    refused = []

    def work(stream, args):
        torch.cuda.set_device(0)
        for i in range(2000):
            if lib.gsa_coo_to_csr(*args) != 0:
                refused.append(L.last_error())
            if i % 200 == 199:
                stream.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not refused
    for io, cols, vo, vals in checks:
        assert np.array_equal(io.cpu().numpy(), cols) and np.array_equal(vo.cpu().numpy(), vals)
