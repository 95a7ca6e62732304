"""The block sampler's 16 x 16 tiling at its edges: ragged sizes, index sets
whose bases share few segments (taken 8 or 4 bases at a time), padded wings,
every weight and kernel option, against the oracle.

Tolerance 1e-12 of the largest entry: sums of at most 144 terms of its size,
a few roundings each, k R < 60."""

import numpy as np
import pytest

from conftest import rel_err
from oracle import block_oracle as BO

from momwire_b200 import accel

pytestmark = pytest.mark.gpu


def _side(rng, n, degree, z0, scattered, mirror=False):
    """n bases on random short segments: runs of neighbours sharing wings, or
    (scattered) wings drawn at random."""
    d1 = degree + 1
    n_seg = n + degree if not scattered else 3 * n + 5
    c = rng.uniform(0.0, 4.0, (n_seg, 3)) + [0.0, 0.0, z0]
    t = rng.standard_normal((n_seg, 3))
    t /= np.linalg.norm(t, axis=1)[:, None]
    h = rng.uniform(0.05, 0.3, n_seg)
    l, r = c - 0.5 * h[:, None] * t, c + 0.5 * h[:, None] * t
    if mirror:
        l, r, t = l * [1, 1, -1], r * [1, 1, -1], t * [1, 1, -1]
    supp = rng.integers(0, n_seg, (n, d1)) if scattered else np.arange(n)[:, None] + np.arange(d1)[None, :]
    polys = rng.standard_normal((n, d1, d1))
    pad = rng.uniform(size=(n, d1)) < 0.1  # the reference pads with segment 0 and zero coefficients
    polys[pad] = 0.0
    supp = np.where(pad, 0, supp)
    return supp, polys, l, r, t, rng.integers(-1, 3, n_seg)


@pytest.mark.parametrize("n_i,n_j,degree,nq,scattered,opt", [
    (1, 1, 2, 4, False, ""), (16, 17, 2, 4, False, ""), (33, 15, 1, 4, False, "ek"), (40, 50, 2, 8, False, "refl"),
    (31, 70, 2, 3, False, "refl ek"), (20, 37, 2, 4, True, ""), (35, 18, 1, 4, True, "refl"), (17, 40, 2, 1, True, "ek")])
def test_block_tiles_match_oracle(n_i, n_j, degree, nq, scattered, opt, cuda_device):
    rng = np.random.default_rng(100 * n_i + n_j)
    I = _side(rng, n_i, degree, 6.0, scattered)
    J = _side(rng, n_j, degree, 1.0, scattered, "refl" in opt)
    t, w = np.polynomial.legendre.leggauss(nq)
    t, w = 0.5 * (t + 1.0), 0.5 * w
    a2, k = 1e-5, 2.0
    om, eps, mu = k * 3e8, 8.85e-12, 1.2566e-6
    base = (*I[:5], *J[:5], a2, k, om, eps, mu, degree, t, w)
    refl = (13.0 - 2.0j, 0.3 + 0.1j, 0.7 - 0.2j)
    if opt == "":
        got = accel.bspline_assemble_offedge_block(*base)
    elif opt == "ek":
        got = accel.bspline_assemble_offedge_block_ek(*base, I[5], J[5], 2e-3)
    elif opt == "refl":
        got = accel.bspline_assemble_offedge_block_refl(*base, *refl)
    else:
        got = accel.bspline_assemble_offedge_block_refl_ek(*base, I[5], J[5], 2e-3, *refl)
    want = BO.offedge_block(*I[:5], *J[:5], a2, k, om, eps, mu, t, w,
                            group=(I[5], J[5]) if "ek" in opt else None, a_ek=2e-3 if "ek" in opt else 0.0,
                            refl=refl if "refl" in opt else None)
    assert got.shape == (n_i, n_j)
    assert rel_err(got, want) < 1e-12
