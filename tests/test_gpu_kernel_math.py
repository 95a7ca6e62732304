"""The kernels' elementary functions over the ranges they claim, against the
correctly rounded values (80-bit arithmetic here).

Bounds, in units in the last place of the result or in u = 2^-53:
  1 / sqrt x  1 ulp, CUDA's own bound for rsqrt: one step of Halley's iteration
              from 20 bits leaves the rounding of 1 - x y^2 (half an ulp) and of
              the last operation;
  sqrt x      0.51 ulp: the residual is exact, its product adds 2^-53 of an ulp's
              order;
  1 / z       4.5 u of |1 / z|: |z|^2 1.5 u, its reciprocal 2 u, the product u;
  sin, cos    2 ulp, CUDA's own bound for sincos (1 ulp is what the series need).
"""

import numpy as np
import pytest

from momwire_b200 import _lib

pytestmark = pytest.mark.gpu
LD = np.longdouble
U = LD(2) ** -53


def _run(which, x, device, y=0.0):
    import torch

    h = np.empty((x.size, 2))
    h[:, 0], h[:, 1] = x, y
    d = torch.from_numpy(h).to(device)
    o = torch.empty_like(d)
    _lib.call("mw_selftest_math", which, x.size, d.data_ptr(), o.data_ptr(), None)
    r = o.cpu().numpy()
    return r[:, 0], r[:, 1]


def _ulps(got, want):
    return np.abs(got.astype(LD) - want) / np.spacing(np.abs(want.astype(float)))


def _spread(rng, n, lo, hi):
    """Mantissas at random, exponents from lo to hi, with the ends and the
    neighbours of powers of two."""
    e = rng.integers(lo, hi + 1, n)
    x = np.ldexp(1.0 + rng.uniform(0, 1, n), e)
    p = np.ldexp(1.0, np.arange(lo, hi + 1))
    return np.concatenate([x, p, np.nextafter(p, np.inf), np.nextafter(p, 0.0)[1:]])


def test_roots(cuda_device):
    x = _spread(np.random.default_rng(1), 200_000, -1021, 1022)
    r, s = _run(0, x, cuda_device)
    root = np.sqrt(x.astype(LD))
    assert _ulps(r, 1 / root).max() <= 1.0
    # (products of x with its inverse root: normal where sqrt x times its
    # rounding errors squared is, as distances squared are)
    ok = (x > 1e-280) & (x < 1e300)
    assert _ulps(s, root)[ok].max() <= 0.51


def test_complex_reciprocal(cuda_device):
    rng = np.random.default_rng(2)
    a = _spread(rng, 100_000, -1019, 1020) * -1.0
    ratio = np.ldexp(rng.uniform(-1, 1, a.size), -rng.integers(0, 60, a.size))
    for x, y in ((a, a * ratio), (a * ratio, a), (a, a), (a, np.zeros_like(a))):
        re, im = _run(1, x, cuda_device, y)
        xs, ys = x.astype(LD), y.astype(LD)
        d = xs * xs + ys * ys
        n = np.hypot(xs / d, ys / d)
        err = np.hypot(re.astype(LD) - xs / d, im.astype(LD) + ys / d)
        assert np.all(err <= 4.5 * U * n + LD(2) ** -1073)  # (components below the normal range round there)


def test_reciprocal_of_special_values_is_the_division(cuda_device):
    tiny = np.array([5e-324, 1e-310, np.ldexp(1.0, -1022), np.inf, -np.inf, np.nan, 0.0])
    x, y = [g.ravel() for g in np.meshgrid(tiny, [0.0, 1e-312])]
    re, im = _run(1, x, cuda_device, y)
    with np.errstate(all="ignore"):  # Smith's quotient 1 / z
        big = np.abs(x) >= np.abs(y)
        r = np.where(big, y / x, x / y)
        den = np.where(big, x + y * r, x * r + y)
        want_re, want_im = np.where(big, 1.0 / den, r / den), np.where(big, -r / den, -1.0 / den)
    assert np.array_equal(np.isnan(re), np.isnan(want_re)) and np.array_equal(np.isnan(im), np.isnan(want_im))
    fin = np.isfinite(want_re) & np.isfinite(want_im)
    assert np.allclose(re[fin], want_re[fin], rtol=1e-9, atol=0) and np.allclose(im[fin], want_im[fin], rtol=1e-9, atol=0)
    assert np.array_equal(np.isinf(re), np.isinf(want_re))


@pytest.mark.parametrize("which,top", [(2, 0.3), (3, 0.75), (4, 40.0)])
def test_phase_steps(which, top, cuda_device):
    rng = np.random.default_rng(which)
    x = np.concatenate([rng.uniform(-top, top, 200_000), [0.0, top, -top, np.nextafter(top, 0), 0.75, -0.75, 1e-300, 5e-9],
                        np.ldexp(rng.uniform(0.5, 1.0, 1000), -rng.integers(0, 60, 1000))])
    x = x[np.abs(x) <= top]
    s, c = _run(which, x, cuda_device)
    xs = x.astype(LD)
    nz = x != 0
    assert _ulps(s[nz], np.sin(xs[nz])).max() <= 2.0 and np.all(s[~nz] == 0)
    assert _ulps(c, np.cos(xs)).max() <= 2.0
