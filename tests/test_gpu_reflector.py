"""The BSOF chain's reflector scalars (bsofi_selftest_reflector) against long
double: beta = -sign(alpha) ||(alpha, x)||, tau = 1 + |alpha| / ||.||, scale =
1 / (alpha - beta), q = -1 / beta.

The bounds are those of the roundings, in units of 2^-53: the squared norm's sum
costs one (half after the square root), every later operation one.
  fast range (squared norm in [2^-930, 2^930)): beta 0.5 + 1; q 1.5 + 1;
    tau (2.5 + 2) / 2; scale 1.5 + 1 (the sum) + 1.
  outside, by rsqrt() (two units) and a division (one): beta 0.5 + 2 + 1; q 2.5;
    tau (2.5 + 2) / 2; scale 3.5 + 1 + 1.
Terms of second order, and the cube of the reciprocal's first error (2^-60), stay
below the tenth of a unit added to each.  Against CUDA's functions, computed
beside them, the two bounds add up.
"""
import numpy as np
import pytest

from bsofi_b200 import _lib

pytestmark = pytest.mark.gpu

U = np.longdouble(2) ** -53
FAST = {"beta": 1.6, "tau": 2.35, "scale": 3.6, "q": 2.6}
RARE = {"beta": 3.6, "tau": 2.35, "scale": 5.6, "q": 2.6}


def _scalars(torch, dev, x2, alpha):
    a, b = torch.from_numpy(x2).to(dev), torch.from_numpy(alpha).to(dev)
    out = torch.empty(len(x2), 7, dtype=torch.float64, device=dev)
    assert _lib.load().bsofi_selftest_reflector(len(x2), a.data_ptr(), b.data_ptr(), out.data_ptr(),
                                                torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _exact(x2, alpha):
    al = alpha.astype(np.longdouble)
    norm = np.sqrt(x2.astype(np.longdouble) + al * al)
    sg = np.copysign(np.longdouble(1), al)
    return {"beta": -sg * norm, "tau": 1 + np.abs(al) / norm, "scale": sg / (np.abs(al) + norm),
            "q": sg / norm}


def _pairs(kind, rng, count=1 << 16):
    m = 1 + rng.random(count)
    if kind == "near one":  # squared norms and pivots of ordinary columns
        return m * 2.0 ** rng.integers(-12, 13, count), rng.standard_normal(count)
    if kind == "any scale":  # pivots from 2^-60 to 2^60 of the norm, norms over the whole range
        e = rng.integers(-940, 941, count) // 2
    elif kind == "low switch":
        e = rng.integers(-468, -462, count)
    else:
        e = rng.integers(462, 468, count)
    lo = rng.integers(-60, 61, count) if kind == "any scale" else rng.integers(-8, 9, count)
    x2 = np.ldexp(m, 2 * e + np.minimum(0, -2 * lo))  # the larger of the two near 2^e
    return x2, np.ldexp(rng.standard_normal(count), e + np.minimum(0, lo))


@pytest.mark.parametrize("kind", ["near one", "any scale", "low switch", "high switch"])
def test_against_long_double(cuda_device, kind):
    import torch
    x2, alpha = _pairs(kind, np.random.default_rng(len(kind)))
    got = _scalars(torch, cuda_device, x2, alpha)
    s2 = x2.astype(np.longdouble) + alpha.astype(np.longdouble) ** 2
    # (At the switch itself either branch may have run.)
    fast = (s2 >= np.longdouble(2) ** -930 * (1 + 4 * U)) & (s2 < np.longdouble(2) ** 930 * (1 - 4 * U))
    assert fast.any() and (kind == "near one" or not fast.all())
    for i, (name, ref) in enumerate(_exact(x2, alpha).items()):
        err = np.abs((got[:, i] - ref) / ref) / U
        assert err[fast].max() <= FAST[name], name
        assert (err[~fast] <= RARE[name]).all(), name
        if i < 3:
            apart = np.abs((got[:, i] - got[:, 4 + i].astype(np.longdouble)) / ref) / U
            assert apart.max() <= FAST[name] + RARE[name], name


def test_nothing_below_the_pivot(cuda_device):
    """LAPACK's H = I: tau = 0, beta = alpha, whatever the pivot."""
    import torch
    alpha = np.array([1.0, -2.5, 0.0, -0.0, 1e300, -1e-300, np.inf, -np.inf])
    got = _scalars(torch, cuda_device, np.zeros(len(alpha)), alpha)
    np.testing.assert_array_equal(got[:, :4], np.stack([alpha, 0 * np.ones(8), np.ones(8), 0 * np.ones(8)], 1))


@pytest.mark.parametrize("x2,alpha", [(np.nan, 1.0), (1.0, np.nan), (np.inf, 1.0)])
def test_what_is_not_a_number_stays_so(cuda_device, x2, alpha):
    import torch
    got = _scalars(torch, cuda_device, np.array([x2]), np.array([alpha]))
    assert np.isnan(got[0, 0])
