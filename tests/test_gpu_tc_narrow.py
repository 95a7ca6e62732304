"""The tensor-core update's epilogue at the edges of its 32-column rounds and
32-row warps: C -= A B against complex128, and nothing outside C written."""

import numpy as np
import pytest

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 48, 64, 65, 96, 129, 255, 257, 288])
@pytest.mark.parametrize("m,k", [(16, 16), (63, 1), (64, 63), (81, 65), (700, 130)])
def test_narrow_update(m, n, k, cuda_device):
    import torch

    lib = _lib.load()
    rng = np.random.default_rng(1000 * m + n)

    def c64(r, c):
        return (rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))).astype(np.complex64)

    A, B, ld = c64(k, m), c64(n, k), m + 3
    Cg = c64(n + 2, ld)  # column-major C in rows 0 .. m-1 of the first n columns
    Ad, Bd, Cd = (torch.from_numpy(x).to(cuda_device) for x in (A, B, Cg))
    wsb = lib.mw_cgemm_tc_workspace_size(m, n, k)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda_device)
    status = torch.zeros(1, dtype=torch.int32, device=cuda_device)
    _lib.call("mw_cgemm_tc_sub", m, n, k, Ad.data_ptr(), m, Bd.data_ptr(), k, Cd.data_ptr(), ld, ws.data_ptr(), wsb,
              status.data_ptr(), None)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got = Cd.cpu().numpy()
    prod = B.astype(np.complex128) @ A.astype(np.complex128)
    want = Cg[:n, :m].astype(np.complex128) - prod
    # the splits leave 2^-21 of each product behind (lo * lo and the lower
    # bits of lo), sums and the final subtraction round in fp32
    bound = (np.abs(B).astype(np.float64) @ np.abs(A).astype(np.float64)) * (2.0**-19 + k * 2.0**-22) \
        + np.abs(want) * 2.0**-22
    assert np.all(np.abs(got[:n, :m] - want) <= bound)
    assert np.array_equal(got[n:], Cg[n:]) and np.array_equal(got[:, m:], Cg[:, m:])
