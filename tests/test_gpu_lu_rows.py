"""The cluster LU with two and three rows to a thread and real interchanges,
and the orders beyond one cluster's rows: random matrices, whose pivots come
from every row that a thread holds.

Batches as in test_gpu_lu_cluster.py.  Large orders on the device: the
factors' residual and the solution's against LAPACK's normwise bounds (a
small multiple of n eps, growth included through |L| and |U|), and every
multiplier at most sqrt 2, which partial pivoting by |re| + |im| gives and a
wrong choice of row would not."""

import numpy as np
import pytest

from test_gpu_lu_cluster import _check, _random, _solve

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


# 160 systems leave a CTA to each: 300 rows are two to a thread, 600 three
@pytest.mark.parametrize("n,nrhs,batch", [(257, 1, 160), (300, 3, 160), (513, 1, 160), (600, 2, 160)])
def test_rows_of_a_thread_compete(n, nrhs, batch, cuda_device):
    A, B = _random((batch, n, n), n), _random((batch, n, nrhs), n + 1)
    LU, ipiv, info, X = _solve(A, B, cuda_device, ldpad=1)
    for b in (0, batch // 3, batch - 1):
        _check(A[b], B[b], LU[b], ipiv[b], info[b], X[b])


# sixteen CTAs: two rows to a thread above 4,096, three above 8,192; beyond
# 12,288 the cooperative panels
@pytest.mark.parametrize("n,nrhs", [(4100, 3), (8200, 2), (12292, 3)])
def test_large_orders(n, nrhs, cuda_device):
    import torch

    g = torch.Generator(device=cuda_device).manual_seed(n)
    A = torch.randn((n, n), dtype=torch.complex128, device=cuda_device, generator=g)  # A[j, i]: entry (i, j)
    B = torch.randn((nrhs, n), dtype=torch.complex128, device=cuda_device, generator=g)
    F, X = A.clone(), B.clone()
    wsb = _lib.load().mw_getrf_workspace_size(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda_device)
    ipiv = torch.zeros(n, dtype=torch.int32, device=cuda_device)
    info = torch.full((2,), 9, dtype=torch.int32, device=cuda_device)
    _lib.call("mw_zgesv", n, nrhs, F.data_ptr(), n, ipiv.data_ptr(), info.data_ptr(), X.data_ptr(), n, ws.data_ptr(),
              wsb, None, None)
    assert info.tolist() == [0, 0]
    r = (X @ A - B).abs().max().item()
    scale = A.abs().sum(0).max().item() * X.abs().max().item() + B.abs().max().item()
    assert r <= 200 * n * EPS * scale
    # rows in the factors' order; L and U transposed like A
    p = np.arange(n)
    moved = 0
    for i, q in enumerate(ipiv.cpu().numpy() - 1):
        assert i <= q < n
        moved += q != i
        p[[i, q]] = p[[q, i]]
    assert moved > 0.99 * (n - 64)
    L = torch.triu(F, 1)
    assert L.abs().max().item() <= np.sqrt(2.0) * (1 + 8 * EPS)
    rowsum = L.abs().sum(0).max().item() + 1.0
    L.diagonal().fill_(1.0)
    U = torch.tril(F)
    umax = U.abs().max().item()
    PA = A[:, torch.from_numpy(p).to(cuda_device)]
    worst = max((PA[c : c + 1024] - U[c : c + 1024] @ L).abs().max().item() for c in range(0, n, 1024))
    assert worst <= 20 * n * EPS * rowsum * umax
