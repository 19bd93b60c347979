"""Conversions on a caller's workspace: it may start on any byte, and not a byte before or after it
is written."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 8, 16, 48, 3])
@pytest.mark.parametrize("kind", ["short", "longer", "long", "one_level"])
@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex128])
def test_conversion_workspace_anywhere(gsa, cuda, dt, kind, shift):
    rng = np.random.default_rng(7)
    m, n, nnz = {"short": (3000, 500, 9000), "longer": (200, 900, 9000), "long": (3, 20_000, 9000),
                 "one_level": (8192 * 4096 + 5, 40, 2000)}[kind]
    r, c = rng.integers(0, m, nnz), rng.integers(0, n, nnz)
    v = rng.integers(1, 99, nnz).astype(dt)
    order = np.lexsort((c, r))  # stable: duplicates keep their order
    lib, L = gsa._lib.load(), gsa._lib
    code = {np.float32: L.F32, np.float64: L.F64, np.complex128: L.C64}[dt]
    need = lib.gsa_coo_to_compressed_workspace_size(0, code, L.IDX32, m, n, nnz)
    arena = torch.full((512 + need + 512,), 0x5a, dtype=torch.uint8, device=cuda)
    first = 256 + shift
    assert arena.data_ptr() % 256 == 0
    t = lambda a: torch.from_numpy(a).to(cuda)
    rd, cd, vd = t((r + 1).astype(np.int32)), t((c + 1).astype(np.int32)), t(v)
    po = torch.zeros(m + 1, dtype=torch.int32, device=cuda)
    io, vo = torch.zeros_like(cd), torch.zeros_like(vd)
    p = lambda a: ctypes.c_void_p(a.data_ptr())
    assert lib.gsa_coo_to_csr(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), code, L.IDX32, m, n, nnz,
                              p(rd), p(cd), p(vd), 1, p(po), p(io), p(vo),
                              ctypes.c_void_p(arena.data_ptr() + first), need) == 0
    assert np.array_equal(po.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]) + 1)
    assert np.array_equal(io.cpu().numpy(), c[order] + 1)
    assert np.array_equal(vo.cpu().numpy(), v[order])
    edge = torch.cat([arena[:first], arena[first + need:]])
    assert bool((edge == 0x5a).all())
