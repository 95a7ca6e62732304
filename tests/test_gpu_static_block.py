"""The diagonal-block factorisation and the rows below it of the static
pivots, at the edges of their 16-column panels, 32-column groups, 8-row warps
and waves of CTAs: the complex64 factors left by mw_zgesv_mixed multiply back
to the matrix, and the solutions agree with numpy."""

import ctypes as C

import numpy as np
import pytest

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu

EPS32 = float(np.finfo(np.float32).eps)


def _solve(Z, B):
    """Factors (numpy complex128), interchanges (0-based), X (device tensor),
    pivoting used, for device tensors Z (n, n) and B (n, nrhs)."""
    import torch

    lib = _lib.load()
    n, nrhs = B.shape
    Zd = Z.T.contiguous()
    Z32 = Zd.to(torch.complex64)
    Bd = B.T.contiguous()
    Xd = torch.empty((nrhs, n), dtype=torch.complex128, device=Z.device)
    ipiv = torch.empty(n, dtype=torch.int32, device=Z.device)
    info = torch.zeros(4, dtype=torch.int32, device=Z.device)
    wsb = lib.mw_zgesv_mixed_workspace_size(n, nrhs)
    ws = torch.empty(wsb, dtype=torch.uint8, device=Z.device)
    it, corr = C.c_int32(0), C.c_double(0.0)
    prev = lib.mw_set_mixed_pivoting(0)
    try:
        _lib.call("mw_zgesv_mixed", n, nrhs, Zd.data_ptr(), n, Z32.data_ptr(), n, ipiv.data_ptr(), Bd.data_ptr(), n,
                  Xd.data_ptr(), n, 1e-10, 10, ws.data_ptr(), wsb, info.data_ptr(), C.byref(it), C.byref(corr), None,
                  None)
    finally:
        lib.mw_set_mixed_pivoting(prev)
    torch.cuda.synchronize()
    return Z32, ipiv.cpu().numpy() - 1, Xd.T, int(lib.mw_last_mixed_pivoting())


def _check_factors(A, F, piv):
    """|L U - P A| <= 8 n eps (|L||U|) entrywise: n products of complex
    numbers, each with up to 2 sqrt(2) roundings, and the final one."""
    n = A.shape[0]
    PA = A.astype(np.complex64).astype(np.complex128)
    for i, p in enumerate(piv):
        if p != i:
            PA[[i, p]] = PA[[p, i]]
    L = np.tril(F, -1) + np.eye(n)
    U = np.triu(F)
    bound = 8 * n * EPS32 * (np.abs(L) @ np.abs(U))
    assert np.all(np.abs(L @ U - PA) <= bound)


def _matrix(n, rng):
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return A + np.eye(n) * (4.0 * np.sqrt(n) + 4.0)


# orders around 16 and 32 columns within the block, then rows below it around
# a warp's eight, the packed operand's 64 and a CTA's share
@pytest.mark.parametrize("n", [2, 15, 16, 17, 31, 33, 48, 80, 97, 112, 113, 127, 128,
                               129, 135, 136, 137, 160, 191, 192, 193, 257, 449, 1500])
def test_factors_multiply_back(n, cuda_device):
    import torch

    rng = np.random.default_rng(n)
    A = _matrix(n, rng)
    B = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    F, piv, X, used = _solve(torch.from_numpy(A).to(cuda_device), torch.from_numpy(B).to(cuda_device))
    assert used == 0
    assert np.array_equal(piv, np.arange(n))
    _check_factors(A, F.cpu().numpy().T.astype(np.complex128), piv)
    want = np.linalg.solve(A, B)
    assert np.linalg.norm(X.cpu().numpy() - want) <= 1e-9 * np.linalg.norm(want)


# a multiplier past the bound: in the first sub-block, below it, in a later
# panel's sub-block, in a partial last block
@pytest.mark.parametrize("n,i,j", [(128, 9, 2), (128, 100, 3), (128, 125, 118), (200, 190, 150)])
def test_large_multiplier_is_interchanged(n, i, j, cuda_device):
    import torch

    rng = np.random.default_rng(n + i)
    A = _matrix(n, rng)
    A[i, j] = 3.0 * A[j, j]
    A[j, i] = 3.0 * A[i, i]
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    F, piv, X, used = _solve(torch.from_numpy(A).to(cuda_device), torch.from_numpy(B).to(cuda_device))
    assert used == 0
    assert piv[j] == i
    _check_factors(A, F.cpu().numpy().T.astype(np.complex128), piv)
    want = np.linalg.solve(A, B)
    assert np.linalg.norm(X.cpu().numpy() - want) <= 1e-9 * np.linalg.norm(want)


def test_rows_beyond_one_wave(cuda_device):
    """13300 rows: the first panels' rows take two waves of CTAs."""
    import torch

    n = 13300
    gen = torch.Generator(device=cuda_device).manual_seed(5)
    A = torch.randn((n, n), dtype=torch.complex128, device=cuda_device, generator=gen)
    A += torch.eye(n, dtype=torch.complex128, device=cuda_device) * (4.0 * n**0.5)
    B = torch.randn((n, 1), dtype=torch.complex128, device=cuda_device, generator=gen)
    _F, piv, X, used = _solve(A, B)
    assert used == 0
    assert np.array_equal(piv, np.arange(n))
    res = torch.linalg.norm(A @ X - B) / torch.linalg.norm(B)
    assert float(res) <= 1e-9


@pytest.mark.parametrize("n", [1795, 1800])
def test_wide_block_rows(n, cuda_device):
    """Block rows of 1,536 columns and more, with interchanges inside the
    blocks (each block's rows reversed): permuted, solved and packed in one
    pass."""
    import torch

    rng = np.random.default_rng(n)
    order = np.concatenate([np.arange(min(b + 128, n) - 1, b - 1, -1) for b in range(0, n, 128)])
    A = _matrix(n, rng)[order]
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    F, piv, X, used = _solve(torch.from_numpy(A).to(cuda_device), torch.from_numpy(B).to(cuda_device))
    assert used == 0
    _check_factors(A, F.cpu().numpy().T.astype(np.complex128), piv)
    want = np.linalg.solve(A, B)
    assert np.linalg.norm(X.cpu().numpy() - want) <= 1e-9 * np.linalg.norm(want)
