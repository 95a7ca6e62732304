"""The fill of a single system with its complex64 copy (fixed order of sums):
the same cases as the fill without one, to the same tolerance, and a copy that
is Z rounded."""

import numpy as np
import pytest

from conftest import rel_err
from oracle import bspline_oracle as O
from test_gpu_fill_paths import CASES

import momwire_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", CASES)
def test_fill_with_copy_matches_oracle(name, cuda_device):
    import torch

    kw = CASES[name]()
    s = momwire_b200.BSplineSolver(**kw, precision="mixed")
    buf = s._alloc()
    s._fill_device(buf, torch.cuda.current_stream(buf["Z"].device).cuda_stream)
    Z = buf["Z"].cpu().numpy().T
    assert rel_err(Z, O.compute_Z(O.make_spec(**kw))) < 1e-11
    assert np.array_equal(buf["Z32"].cpu().numpy().T, Z.astype(np.complex64))
