"""The fill's dispatch: pair quadrature orders, the three phase-series spans
(k times the two segment lengths up to 0.3, up to 0.75, beyond) and the
three block sizes (by the segments a tile may hold), against the oracle.

Tolerance: every entry is a sum of a few hundred terms of the largest
entry's size at most, each with a few units of rounding and of phase error
k R eps (k R < 100): 1e-11 of the largest entry leaves a factor of ten."""

import dataclasses

import numpy as np
import pytest

from conftest import rel_err
from oracle import bspline_oracle as O

import momwire_b200
from momwire_b200 import _tables as T

pytestmark = pytest.mark.gpu

LAM = 20.0


def _parallel(nseg, n_wires=3, **kw):
    wires = [np.array([[2.0 * i, 0.3 * i, 1.0], [2.0 * i, 0.3 * i + 0.1, 9.0 + 0.2 * i]]) for i in range(n_wires)]
    return dict(wires=wires, nsegs=nseg, wavelength=LAM, wire_radius=2e-3, feeds=[(0, None, 1.0)], **kw)


def _brush(n_wires, nseg, **kw):
    """Many one- or two-segment wires from one node: tiles of many segments."""
    rng = np.random.default_rng(n_wires)
    wires = [np.array([[0.0, 0.0, 5.0], [0.0, 0.0, 5.0] + rng.uniform(-1.5, 1.5, 3)]) for _ in range(n_wires)]
    return dict(wires=wires, nsegs=nseg, wavelength=LAM, wire_radius=1e-3,
                junctions=[[(w, "start") for w in range(n_wires)]], feeds=[(0, 0.3, 1.0)], **kw)


CASES = {
    "short_d2": lambda: _parallel(60, degree=2),
    "short_d1_pec": lambda: _parallel(61, degree=1, ground_z=0.0),
    "long_d2": lambda: _parallel(9, degree=2),
    "any_d2": lambda: _parallel(5, degree=2),
    "any_d1_refl": lambda: _parallel(4, degree=1, ground_z=0.0, ground_eps=(13.0, 0.005)),
    "nq1": lambda: _parallel(12, degree=2, n_qp_pair=1),
    "nq3_pec": lambda: _parallel(12, degree=2, n_qp_pair=3, ground_z=0.0),
    "nq5": lambda: _parallel(20, degree=1, n_qp_pair=5),
    "nq8_ek": lambda: _parallel(14, degree=2, n_qp_pair=8, extended_kernel=True),
    "ek_short_pec": lambda: _parallel(60, degree=2, extended_kernel=True, ground_z=0.0),
    "wide_tiles_d2": lambda: _brush(40, 1, degree=2),
    "wide_tiles_pec": lambda: _brush(24, 2, degree=2, ground_z=0.0),
    "mixed_radii": lambda: dict(_parallel(19, degree=2), wire_radius=[1e-3, 3e-3, 1e-3]),
}


@pytest.mark.parametrize("name", CASES)
def test_fill_matches_oracle(name, cuda_device):
    kw = CASES[name]()
    Z = momwire_b200.BSplineSolver(**kw)._compute_Z_operator()
    want = O.compute_Z(O.make_spec(**kw))
    assert rel_err(Z, want) < 1e-11


@pytest.mark.parametrize("name", ["short_d2", "short_d1_pec", "nq3_pec"])
def test_widest_tiles(name, cuda_device):
    """The largest segment count a tile may declare (24) takes the block of
    352 threads, or of 192: the same matrix as with the tiles' own 18."""
    kw = CASES[name]()
    s = momwire_b200.BSplineSolver(**kw)
    t = T.build_tiles(s._basis().supp)
    seg = np.full((t.seg.shape[0], T.MAX_TILE_SEG), -1, dtype=np.int32)
    seg[:, : t.seg.shape[1]] = t.seg
    s._cached_tiles = dataclasses.replace(t, seg=seg, max_seg=T.MAX_TILE_SEG)
    want = momwire_b200.BSplineSolver(**kw)._compute_Z_operator()
    assert np.array_equal(s._compute_Z_operator(), want)
