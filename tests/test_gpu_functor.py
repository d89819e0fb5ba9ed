"""The neighbour functor of pd_test_force against a 64-bit sum over the same cells: the three
lane counts (16 lanes a particle on small systems, four from 75,776 particles on, one from
303,104 on), several layers, sorted and unsorted walks, coinciding particles, a particle
with a NaN coordinate, weights near the largest value of the type.

Tolerance: a term q (x_j - x_i)/r carries a few roundings (u the unit roundoff): the
difference u |dx|, squares and the reciprocal square root some 8 u; summing m terms adds
at most m u of the sum of magnitudes: (m + 10) u sum|q|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _check(pd, dtype, sort, x, q, r, nn, lo, hi, some):
    """pd_test_force on all particles, checked for those listed."""
    n = len(x)
    t = pd.PD_F32 if dtype == F32 else pd.PD_F64
    vd = pd.VectorDist(n, np.full(3, lo), np.full(3, hi), np.zeros(3, np.int32), 0.0, dtype=dtype,
                       props=[(t, 1), (t, 3)])
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, q)
    cl = vd.getCellListGPU(r, opt=pd.CL_NON_SYMMETRIC | (pd.CL_GPU_REORDER if sort else 0), NNIteratorBox=nn)
    vd.updateCellListGPU(cl)
    cs, so = cl.get()
    v = cl.view()
    vd.test_force(cl, 0, 1, sorted=sort)
    if sort:
        vd.restoreOrder(cl, [1])
    got = vd.deviceToHostProp(1).astype(F64)
    cell = np.repeat(np.arange(v.ncells), np.diff(cs))
    where = np.zeros(n, np.int64)
    where[so] = cell
    gs = list(v.gs)
    u = F32(2.0 ** -24) if dtype == F32 else 2.0 ** -53
    for i in some:
        c = where[i]
        c0, c1, c2 = c % gs[0], c // gs[0] % gs[1], c // (gs[0] * gs[1])
        js = []
        for d in range(max(c2 - nn, 0), min(c2 + nn, gs[2] - 1) + 1):
            for b in range(max(c1 - nn, 0), min(c1 + nn, gs[1] - 1) + 1):
                row = gs[0] * (b + gs[1] * d)
                js.append(so[cs[row + max(c0 - nn, 0)]:cs[row + min(c0 + nn, gs[0] - 1) + 1]])
        js = np.concatenate(js)
        d = x[js].astype(F64) - x[i].astype(F64)
        nrm = np.sqrt((d ** 2).sum(1))
        ok = nrm > 1e-6  # (not for a NaN)
        w = q[js].astype(F64)[ok]
        want = (d[ok] / nrm[ok][:, None] * w[:, None]).sum(0)
        assert np.abs(got[i] - want).max() <= (ok.sum() + 10) * u * w.sum()


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("n,r,nn", [(1, 0.3, 1), (37, 0.3, 1), (3001, 0.11, 2), (75776, 0.05, 1), (75775, 0.05, 1)])
def test_functor(pd, dtype, sort, n, r, nn):
    rng = np.random.default_rng(n)
    x = rng.random((n, 3)).astype(dtype)
    if n > 20:
        x[10] = x[11]  # no direction between them: no contribution
    q = (rng.random(n) + 0.5).astype(dtype)
    some = rng.permutation(n)[:300].tolist() + ([10, 11] if n > 20 else [])
    _check(pd, dtype, sort, x, q, r, nn, 0.0, 1.0, some)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("n", [303103, 303104, 303233])
def test_functor_one_lane(pd, dtype, sort, n):
    test_functor(pd, dtype, sort, n, 0.03, 1)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("sort", [False, True])
@pytest.mark.parametrize("n,r", [(3001, 0.11), (80000, 0.05), (303200, 0.03)])
def test_functor_nan_neighbour(pd, dtype, sort, n, r):
    """A particle with a NaN coordinate lies in the cell it is clamped into; no distance to it
    exceeds the limit, so it adds nothing to the sums of the particles beside it."""
    rng = np.random.default_rng(n)
    x = rng.random((n, 3)).astype(dtype)
    x[7] = (np.nan, 0.01, 0.01)
    q = (rng.random(n) + 0.5).astype(dtype)
    beside = np.nonzero((x < 2 * r).all(1))[0].tolist()
    assert len(beside) > 10
    _check(pd, dtype, sort, x, q, r, 1, 0.0, 1.0, beside + [7])


@pytest.mark.parametrize("dtype,q0", [(F32, 1e36), (F64, 1e305)])
@pytest.mark.parametrize("n", [3001, 303200])
def test_functor_large_weights(pd, dtype, q0, n):
    """Weights whose quotient by a distance overflows: the terms q (dx/r) do not."""
    rng = np.random.default_rng(n)
    L = 1e-2
    x = (rng.random((n, 3)) * L).astype(dtype)
    q = ((rng.random(n) + 0.5) * q0).astype(dtype)
    r = L * (3.0 / n) ** (1.0 / 3.0)
    _check(pd, dtype, False, x, q, r, 1, 0.0, L, rng.permutation(n)[:200].tolist())
