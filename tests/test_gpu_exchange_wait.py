"""The bounded wait of the cluster LU's pivot exchange runs out on purpose (a
short limit and rows that never come): it must end with MW_ERR_TIMEOUT and
leave the context usable."""

import ctypes as C
import time

import numpy as np
import pytest

from cases import CASES
from conftest import golden, rel_err

import momwire_b200
from momwire_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [256, 1 << 14])
def test_exchange_wait_times_out_and_context_survives(cuda_device, limit):
    import torch

    lib = _lib.load()
    ws = torch.zeros(16, dtype=torch.uint8, device=cuda_device)
    stream = torch.cuda.current_stream(cuda_device).cuda_stream
    t0 = time.perf_counter()
    st = lib.mw_selftest_wait_timeout(2, limit, C.c_void_p(ws.data_ptr()), C.c_void_p(stream))
    assert st == _lib.MW_ERR_TIMEOUT, lib.mw_last_error()
    assert b"exchange wait gave up" in lib.mw_last_error()
    assert time.perf_counter() - t0 < 30.0
    y = momwire_b200.BSplineSolver(**CASES["config1"]()).compute_port_solution().y
    assert rel_err(y, golden("config1")["y"]) < 1e-10
