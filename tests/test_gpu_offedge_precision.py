"""Precision of the block sampler on far blocks of smooth bases, where the
charges of a basis's wings cancel: against the oracle (both take the phases
at the rounded k R).

Tolerance, in the block's norm: u times the norm of the sums of the terms'
magnitudes.  A term carries about eight roundings of u / sqrt(3) each; the 64
to 144 terms of an entry being independent leaves a third of the tolerance,
moments contracted with cancelling coefficients go past it."""

import numpy as np
import pytest

from conftest import rel_err
from oracle import block_oracle as BO
from test_gpu_offedge_tiles import _side

from momwire_b200 import accel

pytestmark = pytest.mark.gpu

UNIT = {1: [[0, 1], [1, -1]], 2: [[0, 0, 0.5], [0.5, 1, -1], [0.5, -1, 0.5]]}


def _wires(n_wires, n_seg, degree, x0):
    """Parallel half-wave wires from x0 on, their inner B-splines."""
    L = 0.48 * (1 + 0.003 * np.arange(n_wires))
    supp, polys, l, r = [], [], [], []
    for w in range(n_wires):
        h = L[w] / n_seg
        z = -L[w] / 2 + h * np.arange(n_seg + 1)
        p = np.stack([np.full(n_seg + 1, x0 + 0.5 * (w % 2)), np.full(n_seg + 1, 0.5 * (w // 2)), z], 1)
        for j in range(n_seg - degree):
            supp.append(w * n_seg + j + np.arange(degree + 1))
            polys.append(np.array(UNIT[degree]) / h ** np.arange(degree + 1))
        l.append(p[:-1])
        r.append(p[1:])
    l, r = np.vstack(l), np.vstack(r)
    return np.array(supp), np.array(polys), l, r, np.tile([0.0, 0.0, 1.0], (len(l), 1))


def _magnitudes(I, J, a2, k, om, eps, mu, t, w):
    """Per entry, the sum of its terms' magnitudes (parallel wires)."""
    out = 0.0
    nodes = []
    for supp, polys, l, r, _t in (I, J):
        h = np.linalg.norm(r - l, axis=1)[supp]
        u = h[..., None] * t
        e = np.arange(polys.shape[2])
        wl = w * h[..., None]
        f = np.abs((u[..., None] ** e * polys[:, :, None, :]).sum(-1)) * wl
        df = np.abs((e * u[..., None] ** np.maximum(e - 1, 0) * polys[:, :, None, :]).sum(-1)) * wl
        x = (1 - t)[:, None] * l[supp][:, :, None, :] + t[:, None] * r[supp][:, :, None, :]
        n = len(supp)
        nodes.append((f.reshape(n, -1), df.reshape(n, -1), x.reshape(n, -1, 3)))
    (fi, gi, xi), (fj, gj, xj) = nodes
    for q in range(fi.shape[1]):
        for s in range(fj.shape[1]):
            G = 1.0 / (4 * np.pi * np.sqrt(((xi[:, None, q] - xj[None, :, s]) ** 2).sum(-1) + a2))
            out = out + G * (om * mu * fi[:, q, None] * fj[None, :, s] + gi[:, q, None] * gj[None, :, s] / (om * eps))
    return out


@pytest.mark.parametrize("degree", [1, 2])
def test_far_block_keeps_the_terms_precision(degree, cuda_device):
    I, J = _wires(3, 41, degree, 0.0), _wires(4, 41, degree, 3.0)
    t, w = np.polynomial.legendre.leggauss(4)
    t, w = 0.5 * (t + 1.0), 0.5 * w
    a2, k, eps, mu = 2.5e-7, 6.2, 8.8541878188e-12, 1.25663706127e-6
    om = k / np.sqrt(eps * mu)
    got = accel.bspline_assemble_offedge_block(*I, *J, a2, k, om, eps, mu, degree, t, w)
    want = BO.offedge_block(*I, *J, a2, k, om, eps, mu, t, w, group=None, a_ek=0.0, refl=None)
    u = np.finfo(float).eps / 2
    tol = u * np.linalg.norm(_magnitudes(I, J, a2, k, om, eps, mu, t, w))
    assert np.linalg.norm(got - want) < tol


@pytest.mark.parametrize("lo,hi", [(-3.0, 4.0), (2.0, -2.0)])
def test_nodes_off_the_segments(lo, hi, cuda_device):
    """The rule is the caller's: nodes past a segment's ends are integrated
    where they lie, with phase steps up to seven times those of the segments.
    Tolerance as for the tiles, 1e-12 of the largest entry."""
    rng = np.random.default_rng(5)
    I, J = _side(rng, 20, 2, 9.0, False), _side(rng, 18, 2, 0.0, False)
    t, w = np.polynomial.legendre.leggauss(4)
    t = lo + (hi - lo) * 0.5 * (t + 1.0)
    k = 0.45  # |k| times two lengths below 0.3: the shortest series, were it for the lengths alone
    args = (*I[:5], *J[:5], 1e-5, k, k * 3e8, 8.85e-12, 1.2566e-6)
    got = accel.bspline_assemble_offedge_block(*args, 2, t, 0.5 * w)
    want = BO.offedge_block(*args, t, 0.5 * w, group=None, a_ek=0.0, refl=None)
    assert rel_err(got, want) < 1e-12


@pytest.mark.parametrize("n_i,n_j,degree,nq,scattered", [(20, 33, 2, 2, False), (33, 20, 2, 5, False), (18, 35, 1, 6, True),
                                                         (35, 17, 2, 7, True), (4, 60, 1, 5, False)])
def test_every_order_of_the_rule(n_i, n_j, degree, nq, scattered, cuda_device):
    """Stripes of eight observer segments to order 4, of four beyond, with as
    many as the pairs of a round allow.  Tolerance as for the tiles."""
    rng = np.random.default_rng(nq)
    I, J = _side(rng, n_i, degree, 6.0, scattered), _side(rng, n_j, degree, 1.0, scattered)
    t, w = np.polynomial.legendre.leggauss(nq)
    t, w = 0.5 * (t + 1.0), 0.5 * w
    k = 2.0
    args = (*I[:5], *J[:5], 1e-5, k, k * 3e8, 8.85e-12, 1.2566e-6)
    got = accel.bspline_assemble_offedge_block_ek(*args, degree, t, w, I[5], J[5], 2e-3)
    want = BO.offedge_block(*args, t, w, group=(I[5], J[5]), a_ek=2e-3, refl=None)
    assert rel_err(got, want) < 1e-12
