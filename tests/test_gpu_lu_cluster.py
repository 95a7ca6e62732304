"""The complex128 cluster factorisation (mw_zgesv, mw_zgesv_batched) at the
edges of its panels, clusters and rules, against LAPACK.

Tolerances: LAPACK's normwise backward error bound, a small multiple of
n eps; with random matrices of these orders n eps times the growth stays
below 1e-12, and the comparison of solutions adds the condition number."""

import numpy as np
import pytest
import scipy.linalg

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu


def _solve(A, B, device, ldpad=0):
    """(LU, ipiv, info, X) of stacked systems A (b, n, n), B (b, n, m)."""
    import torch

    b, n, m = A.shape[0], A.shape[1], B.shape[2]
    ld = n + ldpad
    Ah = np.zeros((b, n, ld), dtype=np.complex128)
    Ah[:, :, :n] = A.transpose(0, 2, 1)
    Bh = np.full((b, max(m, 1), ld), 7.0, dtype=np.complex128)
    Bh[:, :m, :n] = B.transpose(0, 2, 1)
    Ad, Bd = torch.from_numpy(Ah).to(device), torch.from_numpy(Bh).to(device)
    wsb = _lib.load().mw_getrf_workspace_size(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device=device)
    ipiv = torch.zeros((b, n), dtype=torch.int32, device=device)
    info = torch.full((b, 2), 9, dtype=torch.int32, device=device)
    if b == 1:
        _lib.call("mw_zgesv", n, m, Ad.data_ptr(), ld, ipiv.data_ptr(), info.data_ptr(), Bd.data_ptr(), ld,
                  ws.data_ptr(), wsb, None, None)
    else:
        _lib.call("mw_zgesv_batched", n, m, b, Ad.data_ptr(), ld, n * ld, ipiv.data_ptr(), info.data_ptr(),
                  Bd.data_ptr(), ld, max(m, 1) * ld, ws.data_ptr(), wsb, None, None)
    Xh = Bd.cpu().numpy()
    assert np.all(Xh[:, :, n:] == 7.0)  # nothing written past the rows
    return (Ad.cpu().numpy()[:, :, :n].transpose(0, 2, 1), ipiv.cpu().numpy(), info.cpu().numpy(),
            Xh[:, :m, :n].transpose(0, 2, 1))


def _random(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _check(A, B, LU, ipiv, info, X):
    n = A.shape[0]
    assert list(info) == [0, 0]
    ref, piv = scipy.linalg.lu_factor(A)
    assert np.array_equal(ipiv, piv + 1)
    L, U = np.tril(LU, -1) + np.eye(n), np.triu(LU)
    PA = A.copy()
    for i, p in enumerate(piv):
        PA[[i, p]] = PA[[p, i]]
    eps = np.finfo(float).eps
    assert np.abs(L @ U - PA).max() <= 20 * n * eps * np.abs(L).sum(1).max() * np.abs(U).max()
    if B.shape[1]:
        r = np.abs(A @ X - B).max()
        assert r <= 200 * n * eps * (np.abs(A).sum(1).max() * np.abs(X).max() + np.abs(B).max())


# panel (16), tile (32, 64), warp and cluster edges; the one-launch limit
# (640) and the blocked route with whole and partial last blocks
@pytest.mark.parametrize("n,nrhs", [(1, 1), (2, 0), (15, 3), (16, 1), (17, 17), (31, 2), (32, 65), (33, 64), (63, 1),
                                    (65, 5), (127, 4), (255, 16), (257, 33), (511, 1), (513, 70), (640, 18),
                                    (641, 3), (768, 65), (897, 0), (1300, 40)])
def test_zgesv_matches_lapack(n, nrhs, cuda_device):
    A, B = _random((1, n, n), n), _random((1, n, nrhs), n + 1)
    LU, ipiv, info, X = _solve(A, B, cuda_device, ldpad=n % 3)
    _check(A[0], B[0], LU[0], ipiv[0], info[0], X[0])


@pytest.mark.parametrize("n,nrhs,batch", [(5, 1, 3), (33, 2, 200), (97, 17, 9), (306, 1, 64), (650, 1, 8), (70, 66, 4)])
def test_zgesv_batched_matches_lapack(n, nrhs, batch, cuda_device):
    A, B = _random((batch, n, n), n), _random((batch, n, nrhs), n + 1)
    LU, ipiv, info, X = _solve(A, B, cuda_device, ldpad=1)
    for b in range(0, batch, max(1, batch // 5)):
        _check(A[b], B[b], LU[b], ipiv[b], info[b], X[b])


@pytest.mark.parametrize("n,col", [(40, 0), (40, 33), (700, 650)])
def test_zero_pivot_is_reported(n, col, cuda_device):
    A = np.eye(n, dtype=np.complex128)[None]
    A[0, col, col] = 0.0
    _LU, _ipiv, info, _X = _solve(A, np.ones((1, n, 1), dtype=np.complex128), cuda_device)
    assert info[0][0] == col + 1 and info[0][1] == 0


def test_ties_take_the_first_row(cuda_device):
    """Equal |re| + |im| in a column: LAPACK's izamax takes the first row,
    also after earlier interchanges moved the rows."""
    n = 96
    rng = np.random.default_rng(3)
    A = rng.choice([1.0, -1.0, 1j, -1j], size=(1, n, n)) + 0.0j
    B = _random((1, n, 2), 4)
    LU, ipiv, info, _X = _solve(A, B, cuda_device)
    ref, piv = scipy.linalg.lu_factor(A[0])
    # the first panel's entries are exact in both, so its choices are too
    assert np.array_equal(ipiv[0][:4], piv[:4] + 1)


@pytest.mark.parametrize("scale", [1e-290, 1e290])
def test_extreme_scales(scale, cuda_device):
    """The reciprocal of a pivot neither overflows nor underflows on the way."""
    n = 50
    A, B = _random((1, n, n), 1) * scale, _random((1, n, 1), 2) * scale
    _LU, ipiv, info, X = _solve(A, B, cuda_device)
    assert list(info[0]) == [0, 0]
    want = np.linalg.solve(A[0] / scale, B[0] / scale)
    assert np.abs(X[0] - want).max() <= 1e-11 * np.abs(want).max()
