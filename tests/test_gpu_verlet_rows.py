"""getVerlet / getVerletSym rows against the oracle where the row kernel changes its way:
layers of a tile beyond the shared-memory staging, tiles of more particles than a sweep
takes, coordinates outside the range of the FP32 tests, very small and very large
length scales, the smallest systems."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _positions(kind, n, L, rng):
    x = rng.uniform(0, L, size=(n, 3))
    if kind == "clump":  # most particles within one cell
        x[: 3 * n // 4] = L * 0.4 + rng.uniform(0, 0.02 * L, size=(3 * n // 4, 3))
    elif kind == "line":  # one dense cell row
        x[:, 1:] = L * 0.5 + rng.uniform(0, 0.05 * L, size=(n, 2))
    return x


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("kind,n,scale", [("uniform", 1, 1.0), ("uniform", 33, 1.0), ("uniform", 3001, 1.0),
                                          ("uniform", 2000, 1e-4), ("uniform", 2000, 1e5), ("clump", 4099, 1.0),
                                          ("line", 5003, 1.0)])
def test_rows_equal_the_exact_predicate(pd, orc, dtype, sym, kind, n, scale):
    rng = np.random.default_rng(n + int(sym))
    L, r = 10.0 * scale, (0.9 if kind == "uniform" else 0.6) * scale
    bc = np.ones(3, np.int32)
    lo, hi = np.zeros(3), np.full(3, L)
    x = orc.wrap(_positions(kind, n, L, rng).astype(dtype), lo.astype(dtype), hi.astype(dtype), bc)
    vd = pd.VectorDist(n, lo, hi, bc, r, dtype=dtype)
    vd.hostToDevicePos(x)
    vd.map()
    vd.ghost_get()
    full = vd.deviceToHostPos()
    g = orc.cl_geometry(lo, hi, np.full(3, r), r, dtype=dtype, verlet=True)
    off, idx = orc.verlet(full, n, g, r)
    if sym:
        off, idx = orc.verlet_sym(full, n, off, idx)
    got_off, got = (vd.getVerletSym(r) if sym else vd.getVerlet(r)).get()
    assert np.array_equal(got_off, off)
    assert np.array_equal(got, idx)


@pytest.mark.parametrize("dtype", [F32, F64])
def test_particle_far_outside_the_grid(pd, dtype):
    """Never mapped: it gets an empty row, the others keep theirs."""
    rng = np.random.default_rng(5)
    n, L, r = 1500, 8.0, 1.0
    x = rng.uniform(0, L, size=(n, 3)).astype(dtype)
    x[7] = (1e9, 2.0, 2.0)
    vd = pd.VectorDist(n, np.zeros(3), np.full(3, L), np.zeros(3, np.int32), 0.0, dtype=dtype)
    vd.hostToDevicePos(x)
    off, idx = vd.getVerlet(r).get()
    d = x[:, None].astype(F64) - x[None].astype(F64)
    near = (d ** 2).sum(2)
    sure = np.abs(near - r * r) > 1e-5  # FP32 rounding of d2 near the cutoff
    for i in range(n):
        row = np.zeros(n, bool)
        row[idx[off[i]:off[i + 1]]] = True
        if i == 7:
            assert not row.any()
        else:
            want = near[i] < r * r
            assert np.array_equal(row[sure[i]], want[sure[i]])


@pytest.mark.parametrize("dtype", [F32, F64])
def test_pairs_at_the_cutoff(pd, orc, dtype):
    """Pairs whose distance is r up to a few roundings: many on a jittered shell of each of
    some centres, decided as the exact predicate decides them."""
    rng = np.random.default_rng(23)
    L, r, n = 12.0, 1.3, 6000
    lo, hi, bc = np.zeros(3), np.full(3, L), np.ones(3, np.int32)
    c = rng.uniform(2, L - 2, size=(20, 3))
    u = rng.normal(size=(n, 3))
    u *= (r * (1.0 + rng.integers(-4, 5, size=(n, 1)) * np.finfo(dtype).eps)) / np.linalg.norm(u, axis=1)[:, None]
    x = orc.wrap(np.concatenate([c, c[rng.integers(0, 20, n)] + u]).astype(dtype), lo.astype(dtype),
                 hi.astype(dtype), bc)
    vd = pd.VectorDist(len(x), lo, hi, bc, r, dtype=dtype)
    vd.hostToDevicePos(x)
    vd.map()
    vd.ghost_get()
    g = orc.cl_geometry(lo, hi, np.full(3, r), r, dtype=dtype, verlet=True)
    off, idx = orc.verlet(vd.deviceToHostPos(), len(x), g, r)
    got_off, got = vd.getVerlet(r).get()
    assert np.array_equal(got_off, off)
    assert np.array_equal(got, idx)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("sym", [False, True])
def test_particles_outside_the_grid(pd, dtype, sym):
    """Beyond the padding by a little and by far, close to each other there, infinite, not a
    number of either sign: no row and in no row; all others keep theirs."""
    rng = np.random.default_rng(6)
    n, L, r = 2500, 8.0, 1.0
    x = rng.uniform(0, L, size=(n, 3)).astype(dtype)
    out = {3: (9.6, 4, 4), 4: (9.7, 4, 4), 7: (1e9, 2, 2), 8: (1e9, 2, 2), 9: (-2.5, -2.5, 4), 10: (np.inf, 1, 1),
           11: (1, -np.inf, 1), 12: (np.nan, 7.5, 7.5), 13: (0.2, 0.2, -np.nan), 14: (np.nan, np.nan, np.nan),
           15: (0.1, 0.1, 1e300 if dtype == F64 else 1e38), 16: (0.5, -9.0, 0.5)}
    for i, p in out.items():
        x[i] = p
    x[100:140] = rng.uniform(0, 0.6, size=(40, 3))  # near the border cells that they are clamped into
    x[140:180] = L - rng.uniform(0, 0.6, size=(40, 3))
    vd = pd.VectorDist(n, np.zeros(3), np.full(3, L), np.zeros(3, np.int32), 0.0, dtype=dtype)
    vd.hostToDevicePos(x)
    off, idx = (vd.getVerletSym(r) if sym else vd.getVerlet(r)).get()
    ok = np.ones(n, bool)
    ok[list(out)] = False
    for i in range(n):
        row = np.zeros(n, bool)
        row[idx[off[i]:off[i + 1]]] = True
        if not ok[i]:
            assert not row.any()
            continue
        with np.errstate(over="ignore"):
            d = ((x.astype(F64) - x[i].astype(F64)) ** 2).sum(1)
        want = ok & (np.where(ok, d, 9.0) < r * r)
        if sym:
            want &= np.arange(n) > i
        sure = ~ok | (np.abs(d - r * r) > 1e-5)
        assert np.array_equal(row[sure], want[sure])
