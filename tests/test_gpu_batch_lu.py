"""The batched complex64 factorisation and solve at the edges of their tiles:
panels of 8, 16 and 32 columns with rows in registers (to 512 and 1024 rows)
and in shared memory, block solves of 16, 32 and 64 rows, one to nine
right-hand sides."""

import ctypes as C

import numpy as np
import pytest

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu

EPS32 = float(np.finfo(np.float32).eps)


def _solve(Z, B, device, pw, pad=0):
    """Factors, interchanges (0-based), X of a batch: Z (b, n, n), B (b, n, nr)."""
    import torch

    lib = _lib.load()
    b, n, nr = B.shape
    Zp = np.zeros((b, n, n + pad), dtype=np.complex128)
    Zp[:, :, :n] = Z.transpose(0, 2, 1)
    Zd = torch.from_numpy(Zp).to(device)
    Z32 = Zd.to(torch.complex64)
    Bd = torch.from_numpy(np.ascontiguousarray(B.transpose(0, 2, 1))).to(device)
    Xd = torch.empty((b, nr, n), dtype=torch.complex128, device=device)
    ipiv = torch.empty((b, n), dtype=torch.int32, device=device)
    info = torch.zeros(b, dtype=torch.int32, device=device)
    wsb = lib.mw_zgesv_mixed_batched_workspace_size(n, nr, b)
    ws = torch.empty(wsb, dtype=torch.uint8, device=device)
    it, corr = C.c_int32(0), C.c_double(0.0)
    ld = n + pad
    _lib.call("mw_zgesv_mixed_batched", n, nr, b, pw, Zd.data_ptr(), ld, n * ld, Z32.data_ptr(), ld, n * ld,
              ipiv.data_ptr(), info.data_ptr(), Bd.data_ptr(), n, n * nr, Xd.data_ptr(), 1e-10, 10, ws.data_ptr(), wsb,
              C.byref(it), C.byref(corr), None)
    torch.cuda.synchronize()
    F = Z32.cpu().numpy()[:, :, :n].transpose(0, 2, 1).astype(np.complex128)
    return F, ipiv.cpu().numpy() - 1, Xd.cpu().numpy().transpose(0, 2, 1)


def _permuted(A, piv):
    PA = A.astype(np.complex64).astype(np.complex128)
    for i, p in enumerate(piv):
        if p != i:
            PA[[i, p]] = PA[[p, i]]
    return PA


@pytest.mark.parametrize("pw", [8, 16, 32])
@pytest.mark.parametrize("n,nr,pad", [(1, 1, 0), (7, 2, 1), (15, 3, 0), (17, 1, 0), (31, 5, 0), (33, 1, 3), (63, 9, 0),
                                      (64, 1, 0), (65, 4, 0), (127, 1, 0), (130, 8, 1), (257, 2, 0), (515, 1, 0),
                                      (1030, 3, 0)])
def test_batch_factors_and_solutions(n, nr, pad, pw, cuda_device):
    """Random matrices (interchanges in nearly every column): P A = L U within
    8 n eps |L||U| -- n products of complex numbers, each with up to 2 sqrt 2
    roundings, and the tensor cores' split products, 2^-19 of each -- with
    multipliers of at most 1 in |re| + |im| up to rounding, and X as numpy's."""
    if n * pw * 8 > 200 * 1024:
        pytest.skip("the panel does not fit: refused")
    rng = np.random.default_rng(n + pw)
    b = 3
    Z = rng.standard_normal((b, n, n)) + 1j * rng.standard_normal((b, n, n)) + 0.5 * np.sqrt(n) * np.eye(n)
    B = rng.standard_normal((b, n, nr)) + 1j * rng.standard_normal((b, n, nr))
    F, piv, X = _solve(Z, B, cuda_device, pw, pad)
    for q in range(b):
        L, U = np.tril(F[q], -1) + np.eye(n), np.triu(F[q])
        bound = (8 * n * EPS32 + 2.0**-19) * (np.abs(L) @ np.abs(U))
        assert np.all(np.abs(L @ U - _permuted(Z[q], piv[q])) <= bound)
        # |l| = |a / p| with cabs1(a) <= cabs1(p): at most sqrt 2
        assert np.max(np.abs(np.tril(F[q], -1)), initial=0.0) <= np.sqrt(2) * (1 + 8 * EPS32)
        want = np.linalg.solve(Z[q], B[q])
        assert np.linalg.norm(X[q] - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("n", [40, 600, 1100])
def test_batch_pivot_ties_take_the_first_row(n, cuda_device):
    """Equal candidates in different warps: the lowest row is the pivot."""
    rng = np.random.default_rng(n)
    Z = (1e-3 * rng.standard_normal((1, n, n)) + 4.0 * np.eye(n)).astype(np.complex128)
    Z[0, :, 0] = 0.0
    Z[0, [3, 35, n - 1], 0] = [5.0, -5.0, 5.0j]
    B = np.ones((1, n, 1))
    _F, piv, X = _solve(Z, B.astype(np.complex128), cuda_device, 16)
    assert piv[0, 0] == 3
    want = np.linalg.solve(Z[0], B[0])
    assert np.linalg.norm(X[0] - want) <= 1e-9 * np.linalg.norm(want)


@pytest.mark.parametrize("n", [20, 600, 1100])
def test_batch_zero_column_is_reported(n, cuda_device):
    Z = np.tile(np.eye(n, dtype=np.complex128), (2, 1, 1))
    Z[1, :, 5] = 0.0
    with pytest.raises(Exception, match="matrix 1 of the batch.*column 6"):
        _solve(Z, np.ones((2, n, 1), dtype=np.complex128), cuda_device, 16)
