"""Where the block sampler's results live: ordinary arrays of their own,
through a page-locked buffer of fixed size per thread, whatever their size
against its slots.  Whole values: no tolerance."""

import threading

import numpy as np
import pytest

from blocks import CASES, case

from momwire_b200 import accel

pytestmark = pytest.mark.gpu


def _block(a):
    return accel.bspline_assemble_offedge_block(
        a["supp_I"], a["polys_I"], a["segl_I"], a["segr_I"], a["tan_I"], a["supp_J"], a["polys_J"], a["segl_J"],
        a["segr_J"], a["tan_J"], a["a2"], a["k"], a["omega"], a["eps_"], a["mu_"], a["degree"], a["t"], a["w"])


def test_blocks_are_ordinary_arrays(cuda_device):
    import torch

    a, _want = case("free_d2_far")
    got = _block(a)
    assert not torch.from_numpy(got).is_pinned()
    assert got.flags.owndata and got.flags.writeable and got.flags.c_contiguous
    kept = got.copy()
    _block(case(CASES[0])[0])  # another result through the same buffer
    assert np.array_equal(got, kept)
    with torch.inference_mode():
        assert np.array_equal(_block(a), kept)
    assert np.array_equal(_block(a), kept)


@pytest.mark.parametrize("slots,more", [(0, 0), (0, 1), (0, 1 << 13), (0, (1 << 13) + 1), (1, -1), (1, 0), (1, 1), (2, 7), (5, 0)])
def test_sizes_around_the_slots(slots, more, cuda_device):
    import torch

    from momwire_b200 import _staging

    count = slots * _staging._Bounce.SLOT // 16 + more
    x = torch.randn(count, dtype=torch.complex128, device=cuda_device)
    got = _staging.to_host(torch, torch.cuda.current_stream(cuda_device), x)
    assert got.dtype == np.complex128 and np.array_equal(got, x.cpu().numpy())


def test_threads_do_not_share_slots(cuda_device):
    import torch

    from momwire_b200 import _staging

    bad = []

    def work(seed):
        stream = torch.cuda.Stream(cuda_device)
        with torch.cuda.stream(stream):
            for i in range(8):
                x = torch.full((1_200_000 + 1000 * seed,), float(100 * seed + i), dtype=torch.float64, device=cuda_device)
                if not np.all(_staging.to_host(torch, stream, x) == 100 * seed + i):
                    bad.append(seed)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
