"""The packed port tables a solver keeps between calls are built again when a
setting they depend on has changed, and what building them refuses stays
refused."""

import numpy as np
import pytest

from cases import CASES

import momwire_b200

pytestmark = pytest.mark.gpu


def test_port_grounded_after_a_solve_is_refused(cuda_device):
    s = momwire_b200.BSplineSolver(**CASES["d2_junction_port"]())
    s.compute_port_solution()
    w, end = s.junctions[0][0]
    s.ground_z = float(s.wires_polylines[w][0 if end == "start" else -1][2])
    with pytest.raises(ValueError, match="both grounded and a junction port"):
        s.compute_port_solution()


def test_moved_feed_is_followed(cuda_device):
    kw = CASES["d2_junction_port"]()
    s = momwire_b200.BSplineSolver(**kw)
    s.compute_port_solution()
    w, _arc, v = s.feeds[0]
    s.feeds[0] = (w, 1.25, v)
    fresh = momwire_b200.BSplineSolver(**dict(kw, feeds=[(w, 1.25, v)]))
    assert np.array_equal(s.compute_port_solution().y, fresh.compute_port_solution().y)
