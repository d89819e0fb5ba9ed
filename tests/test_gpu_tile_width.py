"""Automatic tile widths on a system whose densest tiles fit the staging only after the width
was halved several times: a dense rod along x in a box of vapour, long cutoff (88 particles a
cell in the rod, fewer than two on average, so the mean occupancy asks for the widest tile).
The run keeps a width that fits, from one rebuild to the next, and follows the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _rod():
    sp, k = 1.08, (89, 14, 14)
    box = np.array([89 * sp, 110.0, 110.0])
    g = np.stack(np.meshgrid(*[np.arange(c) for c in k], indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(11)
    x = (g + 0.5) * sp + rng.uniform(-0.03, 0.03, size=(len(g), 3)) + [0.0, 45.0, 47.0]
    v = rng.normal(size=x.shape) * 1.5
    return x, v - v.mean(0), box


@pytest.mark.parametrize("mixed", [False, True])
def test_dense_rod_in_a_thin_box(pd, orc, mixed):
    x, v, box = _rod()
    lo, bc, rc, skin, dt, steps = np.zeros(3), np.ones(3, np.int32), 4.5, 0.3, 0.004, 30
    t = pd.PD_F32 if mixed else pd.PD_F64
    vd = pd.VectorDist(len(x), lo, box, bc, rc + skin, dtype=F64, props=[(t, 3), (t, 3)])
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, v.astype(F32 if mixed else F64))
    md = pd.MD(vd, 0, 1, dt=dt, skin=skin, r_cut=rc, precision=pd.PREC_MIXED if mixed else pd.PREC_FP64)
    E = np.concatenate([md.run(k) for k in (1, 14, 15)])
    tx = md.launch_shape()["tile_tx"]
    assert 1 <= tx <= 5  # (5 + 2 cells) * 9 * 88 records of 32 bytes are the most that fit 200 KB
    builds = E[:, 3].sum()
    assert builds >= 2  # the width was chosen again at rebuilds
    _, _, Eo = orc.md_lj(x, v, lo, box, bc, rc + skin, rc, skin, 1.0, 1.0, dt, 1.0, steps)
    if mixed:
        tot, toto = E[:, 0] + E[:, 1], Eo[1:, 0] + Eo[1:, 1]
        assert np.max(np.abs(tot - toto) / np.abs(toto)) < 2e-5
    else:
        np.testing.assert_allclose(E[:, :3], Eo[1:, :3], rtol=1e-9)


@pytest.mark.parametrize("form", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("tx", [0, 4])
def test_tiles_outgrow_the_last_sizes(pd, orc, form, tx):
    """A build takes the sizes of the one before with a margin of an eighth and 32 records. Here each
    step pulls the particles together by a tenth of their distance from the centre, so that the rows
    and tiles grow by more than a third from one build to the next, and the build is made again."""
    k, sp, dt, steps = 20, 1.4, 0.01, 4
    L = k * sp
    rng = np.random.default_rng(2)
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = (g + 0.5) * sp + rng.uniform(-0.05, 0.05, size=(k ** 3, 3))
    v = -(x - L / 2) * (0.1 / dt)
    dtype = F32 if form == "f32" else F64
    t = pd.PD_F64 if form == "f64" else pd.PD_F32
    lo, box, bc = np.zeros(3), np.full(3, L), np.ones(3, np.int32)
    vd = pd.VectorDist(len(x), lo, box, bc, 2.8, dtype=dtype, props=[(t, 3), (t, 3)])
    vd.hostToDevicePos(x.astype(dtype))
    vd.hostToDeviceProp(0, v)
    md = pd.MD(vd, 0, 1, dt=dt, skin=0.3, sigma=0.3, precision=pd.PREC_MIXED if form == "mixed" else pd.PREC_FP64)
    md.set_tiles(True, tx)
    md.run(0)
    E, rows = [], [md.stats()[1]]
    for _ in range(steps):
        E.append(md.run(1))
        rows.append(md.stats()[1])
    E = np.concatenate(E)
    assert all(b > 1.3 * a for a, b in zip(rows, rows[1:]))
    xo, _, Eo = orc.md_lj(x, v, lo, box, bc, 2.8, 2.5, 0.3, 1.0, 0.3, dt, 1.0, steps)
    assert np.array_equal(E[:, 3], np.ones(steps))
    if form == "f64":
        np.testing.assert_allclose(E[:, :3], Eo[1:, :3], rtol=1e-9)
    else:
        tot, toto = E[:, 0] + E[:, 1], Eo[1:, 0] + Eo[1:, 1]
        assert np.max(np.abs(tot - toto) / np.abs(toto)) < 2e-5
    off, idx, tiled = md.verlet()
    assert tiled
    allp = vd.deviceToHostPos()
    if form == "f64":
        G = orc.cl_geometry(lo, box, 2.8, 2.8, verlet=True)
        eoff, _ = orc.verlet(allp, len(x), G, 2.8)
        assert np.array_equal(np.diff(off), np.diff(eoff))
