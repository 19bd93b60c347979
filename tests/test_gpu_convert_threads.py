"""Host threads that convert matrices of different sizes at once: no call refuses another's launch.
Buckets of 5000 entries take 100 KB of shared memory, those of the small matrices less than 48 KB."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
def test_conversions_at_once(gsa, cuda, dt):
    mats, wants = [], []
    for t, (n, nnz) in enumerate([(100, 500_000), (1500, 20_000), (100, 500_000), (1500, 20_000), (2000, 30_000),
                                  (60, 300_000), (3000, 9000), (1500, 20_000)]):
        rng = np.random.default_rng(t)
        r, c, v = rng.integers(0, n, nnz), rng.integers(0, n, nnz), rng.integers(1, 99, nnz).astype(dt)
        mats.append(gsa.adapt(cuda, gsa.GenericSparseMatrixCOO(n, n, (r + 1).astype(np.int32), (c + 1).astype(np.int32), v)))
        order = np.lexsort((c, r))
        wants.append(((c[order] + 1).astype(np.int32), v[order]))
    wrong = []

    def work(A, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(1000):
                    X = gsa.GenericSparseMatrixCSR(A)
                    if i % 250 == 249 and not (np.array_equal(X.colval.cpu().numpy(), want[0]) and
                                               np.array_equal(X.nzval.cpu().numpy(), want[1])):
                        wrong.append("result")
        except Exception as e:
            wrong.append(str(e))
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in zip(mats, wants)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
