"""Arrays at the alignment of their doubles and floats, not of their complex
entries: the C interface takes them.  The fills, the block sampler and the
Sommerfeld remainder give the bits they give on aligned arrays (the same
operations, stored in two pieces); factorisations and solves are held to
LAPACK's normwise bounds; mw_zgesv and mw_zgesv_batched refuse."""

import ctypes as C

import numpy as np
import pytest
import scipy.linalg

from blocks import case
from test_gpu_fill_paths import CASES
from test_gpu_somm_q_tiles import _structure

import momwire_b200
from momwire_b200 import _lib

pytestmark = pytest.mark.gpu


def _off(torch, count, dtype, off, device):
    """`count` zeros, `off` scalars past an aligned address."""
    buf = torch.zeros(count + 4, dtype=dtype, device=device)
    assert buf.data_ptr() % 16 == 0
    return buf[off : off + count]


@pytest.mark.parametrize("name", ["long_d2", "any_d1_refl", "nq3_pec"])
@pytest.mark.parametrize("copy", [False, True], ids=["z", "z32"])
def test_fill(name, copy, cuda_device):
    import torch

    s = momwire_b200.BSplineSolver(**CASES[name]())
    dt, n, nm = s._dev_tables(), s._basis().n, s.degree + 1
    fr, g = _lib.Freq(float(s.k), float(s.omega), float(s.eps), float(s.mu)), s._ground_struct()
    out = []
    for off in (0, 1):
        table = _off(torch, dt.table_rows * nm * nm * 2, torch.float64, off, cuda_device)
        Z = _off(torch, 2 * n * n, torch.float64, off, cuda_device)
        z32 = _off(torch, 2 * n * n, torch.float32, off, cuda_device)
        p32 = z32.data_ptr() if copy else None
        _lib.call("mw_same_edge_table", C.byref(dt.edges), s.degree, s.n_qp_pair, 0, float(s.k), table.data_ptr(), None)
        _lib.call("mw_fill_z", C.byref(dt.seg), C.byref(dt.basis), table.data_ptr(), C.byref(dt.edges), C.byref(fr),
                  s.n_qp_pair, Z.data_ptr(), n, p32, n, None)
        if g is not None:
            _lib.call("mw_fill_z_image", C.byref(dt.seg), C.byref(dt.basis), C.byref(g), C.byref(fr), s.n_qp_pair,
                      Z.data_ptr(), n, p32, n, None)
        out.append((Z.cpu().numpy(), z32.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0]).max() > 0


def test_batched_fill(cuda_device):
    import torch

    s = momwire_b200.BSplineSolver(**CASES["nq3_pec"]())
    dt, n, nm = s._dev_tables(), s._basis().n, s.degree + 1
    kd = torch.tensor([[s.k, 1.1 * s.k], [s.omega, 1.1 * s.omega]], dtype=torch.float64, device=cuda_device)
    out = []
    for off in (0, 1):
        table = _off(torch, 2 * dt.table_rows * nm * nm * 2, torch.float64, off, cuda_device)
        Z = _off(torch, 4 * n * n, torch.float64, off, cuda_device)
        z32 = _off(torch, 4 * n * n, torch.float32, off, cuda_device)
        _lib.call("mw_fill_z_batch", C.byref(dt.seg), C.byref(dt.basis), C.byref(dt.edges), 2, kd[0].data_ptr(),
                  kd[1].data_ptr(), float(s.eps), float(s.mu), s.n_qp_pair, 0, 0.0, 1, table.data_ptr(), Z.data_ptr(),
                  n, n * n, z32.data_ptr(), n, n * n, None)
        out.append((Z.cpu().numpy(), z32.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_sommerfeld_remainder(cuda_device):
    import torch

    s = momwire_b200.BSplineSolver(**_structure(3, 17, 2, 3))
    dt, n = s._dev_tables(), s._basis().n
    grid = s._somm_grid(0)
    out = []
    for off in (0, 1):
        Z = _off(torch, 2 * n * n, torch.float64, off, cuda_device)
        z32 = _off(torch, 2 * n * n, torch.float32, off, cuda_device)
        _lib.call("mw_somm_remainder_q", C.byref(dt.seg), C.byref(dt.basis), C.byref(grid), 3, 0.0, float(s.k),
                  Z.data_ptr(), n, z32.data_ptr(), n, None)
        out.append((Z.cpu().numpy(), z32.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_block(cuda_device):
    import torch

    a, _want = case("free_d2")
    keep, sides = [], []
    for x in "IJ":
        t = [torch.from_numpy(np.ascontiguousarray(a[f"{f}_{x}"].astype(np.int32 if f == "supp" else np.float64)))
             .to(cuda_device) for f in ("supp", "polys", "segl", "segr", "tan")]
        keep.append(t)
        sides.append(_lib.BlockSide(t[0].shape[0], t[0].data_ptr(), t[1].data_ptr(), t[2].shape[0], t[2].data_ptr(),
                                    t[3].data_ptr(), t[4].data_ptr(), None))
    nI, nJ = sides[0].n_basis, sides[1].n_basis
    fr = _lib.Freq(a["k"], a["omega"], a["eps_"], a["mu_"])
    t, w = np.ascontiguousarray(a["t"]), np.ascontiguousarray(a["w"])
    out = []
    for off in (0, 1):
        Z = _off(torch, 2 * nI * nJ, torch.float64, off, cuda_device)
        _lib.call("mw_offedge_block", a["degree"], C.byref(sides[0]), C.byref(sides[1]), a["a2"], C.byref(fr), t.size,
                  t.ctypes.data, w.ctypes.data, None, 0.0, Z.data_ptr(), nJ, None)
        out.append(Z.cpu().numpy())
    assert np.array_equal(*out)


@pytest.mark.parametrize("n", [21, 100, 300])
@pytest.mark.parametrize("offs", [(1, 1), (1, 0), (0, 1)])
def test_factor_and_solve(n, offs, cuda_device):
    import torch

    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    B = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    Ad, Bd = (_off(torch, 2 * m.size, torch.float64, o, cuda_device) for m, o in zip((A, B), offs))
    for d, m in ((Ad, A), (Bd, B)):
        d.copy_(torch.from_numpy(np.ascontiguousarray(m.T).view(np.float64).ravel()))
    wsb = _lib.load().mw_getrf_workspace_size(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda_device)
    ipiv = torch.zeros(n, dtype=torch.int32, device=cuda_device)
    info = torch.full((2,), 9, dtype=torch.int32, device=cuda_device)
    _lib.call("mw_zgetrf", n, Ad.data_ptr(), n, ipiv.data_ptr(), info.data_ptr(), ws.data_ptr(), wsb, None, None)
    assert info.tolist() == [0, 0]
    _lu, piv = scipy.linalg.lu_factor(A)
    assert np.array_equal(ipiv.cpu().numpy(), piv + 1)
    _lib.call("mw_zgetrs", n, 3, Ad.data_ptr(), n, ipiv.data_ptr(), Bd.data_ptr(), n, None)
    X = Bd.cpu().numpy().view(np.complex128).reshape(3, n).T
    eps = np.finfo(float).eps
    assert np.abs(A @ X - B).max() <= 200 * n * eps * (np.abs(A).sum(1).max() * np.abs(X).max() + np.abs(B).max())


def test_one_call_solves_refuse(cuda_device):
    import torch

    n = 8
    lib = _lib.load()
    ws = torch.empty(lib.mw_getrf_workspace_size(n), dtype=torch.uint8, device=cuda_device)
    A, B = (_off(torch, 2 * n * n, torch.float64, 0, cuda_device) for _ in range(2))
    ip = torch.zeros(n, dtype=torch.int32, device=cuda_device)
    for a, b in ((8, 0), (0, 8)):
        args = (ip.data_ptr(), ip.data_ptr(), B.data_ptr() + b)
        assert lib.mw_zgesv(n, 1, A.data_ptr() + a, n, *args, n, ws.data_ptr(), ws.numel(), None,
                            None) == _lib.MW_ERR_INVALID
        assert b"16-byte aligned" in lib.mw_last_error()
        assert lib.mw_zgesv_batched(n, 1, 1, A.data_ptr() + a, n, n * n, *args, n, n, ws.data_ptr(), ws.numel(), None,
                                    None) == _lib.MW_ERR_INVALID


def test_mixed_batch(cuda_device):
    """Z32 at the alignment of its floats: the batched factors are read in
    two pieces, to the same solution."""
    import torch

    n, m, b = 150, 2, 5
    g = torch.Generator(device=cuda_device).manual_seed(7)
    Z = torch.randn((b, n, n), dtype=torch.complex128, device=cuda_device, generator=g)
    Z += 30.0 * torch.eye(n, dtype=torch.complex128, device=cuda_device)
    B = torch.randn((m, n), dtype=torch.complex128, device=cuda_device, generator=g)
    lib = _lib.load()
    wsb = lib.mw_zgesv_mixed_batched_workspace_size(n, m, b)
    out = []
    for off in (0, 1):
        z32 = _off(torch, 2 * b * n * n, torch.float32, off, cuda_device)
        z32.copy_(torch.view_as_real(Z.to(torch.complex64)).reshape(-1))
        X = torch.empty((b, m, n), dtype=torch.complex128, device=cuda_device)
        ipiv = torch.empty((b, n), dtype=torch.int32, device=cuda_device)
        info = torch.zeros(b, dtype=torch.int32, device=cuda_device)
        ws = torch.empty(wsb, dtype=torch.uint8, device=cuda_device)
        it, corr = C.c_int32(0), C.c_double(0.0)
        _lib.call("mw_zgesv_mixed_batched", n, m, b, 16, Z.data_ptr(), n, n * n, z32.data_ptr(), n, n * n,
                  ipiv.data_ptr(), info.data_ptr(), B.data_ptr(), n, 0, X.data_ptr(), 1e-10, 20, ws.data_ptr(), wsb,
                  C.byref(it), C.byref(corr), None)
        out.append(X.cpu().numpy())
    assert np.array_equal(*out)
