"""The Sommerfeld remainder's tiling: every observer-node chunking (orders 1,
3, 4, 5, 8), both degrees, short wires and tile remainders, against the
same node-to-node projections integrated in numpy.

Tolerance 1e-12 of the largest entry: sums of at most (d+1)^2 n_qp^2 terms
of its size."""

import numpy as np
import pytest

from conftest import rel_err

import momwire_b200

pytestmark = pytest.mark.gpu

LAM = 10.0


def _structure(n_wires, nseg, degree, n_qp):
    rng = np.random.default_rng(10 * n_wires + nseg)
    wires = []
    for _ in range(n_wires):
        p = rng.uniform([0.0, 0.0, 1.0], [6.0, 6.0, 4.0])
        d = rng.standard_normal(3)
        q = p + 0.8 * d / np.linalg.norm(d)
        q[2] = abs(q[2]) + 0.2
        wires.append(np.array([p, q]))
    return dict(wires=wires, nsegs=nseg, degree=degree, wavelength=LAM, wire_radius=1e-3, ground_z=0.0,
                ground_eps=(13.0, 0.005), ground_model="sommerfeld", feeds=[(0, None, 1.0)],
                n_qp_sommerfeld=n_qp)


@pytest.mark.parametrize("n_wires,nseg,degree,n_qp", [(1, 5, 2, 3), (9, 2, 2, 3), (2, 41, 2, 3), (3, 17, 1, 1),
                                                     (5, 7, 2, 4), (3, 20, 2, 5), (4, 9, 1, 8), (20, 1, 2, 3)])
def test_remainder_matches_node_projections(n_wires, nseg, degree, n_qp, cuda_device):
    import ctypes as C

    import torch

    from momwire_b200 import _lib

    s = momwire_b200.BSplineSolver(**_structure(n_wires, nseg, degree, n_qp))
    st = torch.cuda.current_stream().cuda_stream
    dt, n = s._dev_tables(), s._basis().n
    grid = s._somm_grid(st)
    Z = torch.zeros((n, n), dtype=torch.complex128, device=cuda_device)
    z32 = torch.zeros((n, n), dtype=torch.complex64, device=cuda_device)
    _lib.call("mw_somm_remainder_q", C.byref(dt.seg), C.byref(dt.basis), C.byref(grid), n_qp, 0.0, float(s.k),
              Z.data_ptr(), n, z32.data_ptr(), n, st)
    got = -Z.cpu().numpy().T
    assert np.array_equal(z32.cpu().numpy(), Z.cpu().numpy().astype(np.complex64))
    geom, basis = s._geometry(), s._basis()
    t, w = np.polynomial.legendre.leggauss(n_qp)
    t, w = 0.5 * (t + 1.0), 0.5 * w
    nodes = geom.seg_l[:, None, :] + t[None, :, None] * (geom.seg_r - geom.seg_l)[:, None, :]
    obs = torch.from_numpy(np.ascontiguousarray(nodes.reshape(-1, 3))).to(cuda_device)
    tan = torch.from_numpy(np.ascontiguousarray(np.repeat(geom.tangents, n_qp, 0))).to(cuda_device)
    F = torch.empty((obs.shape[0], obs.shape[0]), dtype=torch.complex128, device=cuda_device)
    _lib.call("mw_somm_field_proj", obs.shape[0], obs.data_ptr(), tan.data_ptr(), obs.shape[0], obs.data_ptr(),
              tan.data_ptr(), 0.0, float(s.k), C.byref(grid), F.data_ptr(), st)
    phi = np.zeros((n, geom.n, n_qp))
    u = geom.h[:, None] * t
    for a in range(degree + 1):
        m = np.flatnonzero(basis.supp[:, a] >= 0)
        sg = basis.supp[m, a]
        pw = u[sg][..., None] ** np.arange(degree + 1)
        np.add.at(phi, (m, sg), np.einsum("mqp,mp->mq", pw, basis.polys[m, a]) * (w * geom.h[sg][:, None]))
    phi = phi.reshape(n, -1)
    assert rel_err(got, phi @ F.cpu().numpy() @ phi.T) < 1e-12
