"""The neighbour functor's reciprocal square root (binomial series on the hardware approximation)
against 1/sqrt(x) in a longer type, over the squared distances that it is used for: from 1e-12 to
the largest number.

Bound: with u the unit roundoff, e = 1 - (x y) y carries the rounding of x y, u at most (x y^2 is 1 to
2^-19), and its own, far less; half of it reaches the result. The series left out is below u / 8,
the last operation rounds by u: (1 + 1/2 + 1/8 + 1/8) u relative, 1.75 u."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rsqrt_error_bound(dtype):
    from openfpm_pdata_b200 import pd
    rng = np.random.default_rng(5)
    f = np.finfo(dtype)
    lo, hi = np.log2(1e-12), np.log2(float(f.max)) - 1e-3
    exps = np.exp2(np.arange(np.ceil(lo), np.floor(hi)))
    x = np.concatenate([np.exp2(rng.uniform(lo, hi, 400000)), np.exp2(rng.uniform(lo, 8, 400000)),
                        np.linspace(0.25, 4.0, 200001), exps, np.nextafter(exps.astype(dtype), dtype(0)),
                        [float(f.max)]]).astype(dtype)
    got = pd.selftest_rsqrt(x).astype(np.longdouble)
    want = 1 / np.sqrt(x.astype(np.longdouble))
    err = np.abs(got / want - 1)
    assert err.max() <= 1.75 * float(f.eps) / 2, (err.max() / (float(f.eps) / 2), x[err.argmax()])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rsqrt_of_an_overflowed_square(dtype):
    from openfpm_pdata_b200 import pd
    got = pd.selftest_rsqrt(np.array([np.inf, np.nan, 1.0], dtype))
    assert got[0] == 0 and np.isnan(got[1]) and got[2] == 1
