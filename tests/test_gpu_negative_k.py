"""A negative wavenumber, the other time convention: with k and omega both
negated the kernel and the 1 / (j omega eps) term are conjugated, so lossless
blocks, matrices and admittances are the conjugates of the positive ones.

Segments long enough (|k| times two lengths up to 2 in the block, to 5 in the
fills) that the series for short phase steps would be visibly wrong.
Tolerance: the same operations with mirrored signs, 1e-12 of the largest
entry; the admittances add the condition number of a few hundred."""

import numpy as np
import pytest

from conftest import rel_err
from test_gpu_fill_paths import CASES
from test_gpu_offedge_tiles import _side

import momwire_b200
from momwire_b200 import accel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,ek", [(1, False), (2, True), (2, False)])
def test_block_of_negative_k_is_the_conjugate(degree, ek, cuda_device):
    rng = np.random.default_rng(degree)
    I, J = _side(rng, 20, degree, 6.0, False), _side(rng, 23, degree, 1.0, False)
    t, w = np.polynomial.legendre.leggauss(4)

    def block(sign):
        k = sign * 4.0
        base = (*I[:5], *J[:5], 1e-5, k, k * 3e8, 8.85e-12, 1.2566e-6, degree, 0.5 * (t + 1.0), 0.5 * w)
        if ek:
            return accel.bspline_assemble_offedge_block_ek(*base, I[5], J[5], 2e-3)
        return accel.bspline_assemble_offedge_block(*base)

    assert rel_err(block(-1), block(1).conj()) < 1e-12


@pytest.mark.parametrize("name", ["long_d2", "any_d2", "nq3_pec"])
def test_fills_of_negative_k_are_the_conjugates(name, cuda_device):
    kw = CASES[name]()
    s = momwire_b200.BSplineSolver(**kw)
    k = np.array([4.0, 5.0]) * s.k
    assert rel_err(s.compute_y_matrix_swept(-k), s.compute_y_matrix_swept(k).conj()) < 1e-10
    # Z beside its complex64 copy (the mixed route's fill)
    m = momwire_b200.BSplineSolver(**kw, precision="mixed")
    buf = m._alloc()
    z = []
    for sign in (1, -1):
        with m._k_restored():
            m._set_k(sign * k[0])
            m._fill_device(buf, 0)
        z.append((buf["Z"].cpu().numpy().copy(), buf["Z32"].cpu().numpy().copy()))
    assert rel_err(z[1][0], z[0][0].conj()) < 1e-12
    assert rel_err(z[1][1], z[0][1].conj()) < 1e-6
