"""A cancellation flag raised while a batch of FP64 systems is being solved."""

import threading
import time

import numpy as np
import pytest

from cases import CASES

import momwire_b200
from momwire_b200 import CancelToken, SolveAborted, _lib

pytestmark = pytest.mark.gpu


def _batch(n, batch, cuda_device, token=None, raise_after=None):
    """Seconds of one mw_zgesv_batched call until the device is done, the
    status it raised, and X; the flag is raised `raise_after` seconds after
    the call's start."""
    import torch

    g = torch.Generator(device=cuda_device).manual_seed(n)
    A = torch.randn((batch, n, n), dtype=torch.complex128, device=cuda_device, generator=g)
    B = torch.randn((batch, 2, n), dtype=torch.complex128, device=cuda_device, generator=g)
    wsb = _lib.load().mw_getrf_workspace_size(n)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda_device)
    ipiv = torch.zeros((batch, n), dtype=torch.int32, device=cuda_device)
    info = torch.zeros((batch, 2), dtype=torch.int32, device=cuda_device)
    torch.cuda.synchronize()
    timer = threading.Timer(raise_after, token.cancel) if raise_after else None
    t0, status = time.perf_counter(), 0
    if timer:
        timer.start()
    try:
        _lib.call("mw_zgesv_batched", n, 2, batch, A.data_ptr(), n, n * n, ipiv.data_ptr(), info.data_ptr(),
                  B.data_ptr(), n, 2 * n, ws.data_ptr(), wsb, token.ptr if token else None, None)
    except _lib.NativeError as e:
        status = e.status
    torch.cuda.synchronize()
    if timer:
        timer.join()
    return time.perf_counter() - t0, status, B


def test_flag_stops_a_batch_between_its_launches(cuda_device):
    n, batch = 1000, 300  # some 65 ms in five launches
    _batch(n, batch, cuda_device)
    full, status, X = _batch(n, batch, cuda_device)
    assert status == 0
    _t, status, _X = _batch(n, batch, cuda_device, CancelToken(), raise_after=0.2 * full)
    assert status == _lib.MW_ERR_CANCELLED
    # an unraised flag changes nothing but the launches
    _t, status, Y = _batch(n, batch, cuda_device, CancelToken())
    assert status == 0 and np.array_equal(X.cpu().numpy(), Y.cpu().numpy())


def test_flag_raised_in_a_sweeps_last_batch_aborts(cuda_device, monkeypatch):
    token = CancelToken()
    s = momwire_b200.BSplineSolver(**CASES["config1"](), cancel=token)
    ks = np.linspace(0.9 * s.k, 1.1 * s.k, 12)
    s.compute_y_matrix_swept(ks)
    real = _lib.call

    def call(name, *args):
        real(name, *args)
        if name == "mw_zgesv_batched":
            token.cancel()  # all of the sweep's work is enqueued

    monkeypatch.setattr(_lib, "call", call)
    with pytest.raises(SolveAborted):
        s.compute_y_matrix_swept(ks)
