"""The cell-list driver's bucket kernel against the FP64 oracle: the smallest systems, a box
of few cells, open boundaries, FP32 storage, a dense corner of an empty box.  A run equals
runs of one step and a second identical run bit for bit (the order in which buckets fill does
not matter).  The one-cluster kernel that it hands over to where a bucket overflows: from the
first step, after an odd and after an even number of steps; and by itself in a box of too many
cells for buckets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _md(pd, x, v, L, bc, dtype, dt=0.002):
    t = pd.PD_F64 if dtype == F64 else pd.PD_F32
    vd = pd.VectorDist(x.shape[0], np.zeros(3), np.full(3, L), np.asarray(bc, np.int32), 2.5, dtype=dtype,
                       props=[(t, 3), (t, 3), (pd.PD_I32, 1)])
    vd.hostToDevicePos(x.astype(dtype))
    vd.hostToDeviceProp(0, v)
    vd.hostToDeviceProp(2, np.arange(x.shape[0]))
    return vd, pd.MD(vd, 0, 1, dt=dt, skin=0.0, use_cell_list=True)


def _by_id(vd):
    i = vd.deviceToHostProp(2, with_ghost=False)
    x, v = vd.deviceToHostPos(with_ghost=False), vd.deviceToHostProp(0, with_ghost=False)
    xo, vo = np.empty_like(x), np.empty_like(v)
    xo[i], vo[i] = x, v
    return xo, vo


def _system(kind):
    from openfpm_pdata_b200 import workloads
    if kind == "one":
        return np.array([[1.0, 7.9, 0.1]]), np.array([[3.0, 2.0, -4.0]]), 8.0
    if kind == "clump":  # 1728 particles in a corner of a box of 60: up to 27 a cell there, 0.1 on average
        x, v, _ = workloads.lj_lattice(12, 0.98, 0.03, seed=4)
        return x + 0.5, v * 0.3, 60.0
    side, sp = {"few cells": (8, 1.02), "c1": (16, 1.0), "many": (33, 1.05)}[kind]
    return workloads.lj_lattice(side, sp, 0.05, seed=5)


@pytest.mark.parametrize("kind", ["one", "few cells", "c1", "many", "clump"])
def test_follows_the_oracle(pd, orc, kind):
    x, v, L = _system(kind)
    steps = 6 if kind == "many" else 25
    lo, hi, bc = np.zeros(3), np.full(3, L), np.ones(3, np.int32)
    vd, md = _md(pd, x, v, L, bc, F64)
    E = np.concatenate([md.run(2), md.run(steps - 2)])
    xo, vo, Eo = orc.md_lj(x, v, lo, hi, bc, 2.5, 2.5, 0.0, 1.0, 1.0, 0.002, 1.0, steps)
    np.testing.assert_allclose(E[:, :3], Eo[1:, :3], rtol=1e-9, atol=1e-9)
    gx, gv = _by_id(vd)
    d = gx - xo
    d -= L * np.round(d / L)
    assert np.abs(d).max() < 1e-9
    # the images belong to the last positions, with their properties
    n = vd.size_local()
    pos = vd.deviceToHostPos()
    img, src, _ = orc.ghost_get(pos[:n], lo, hi, bc, 2.5)
    assert np.array_equal(pos[n:], img)
    assert np.array_equal(vd.deviceToHostProp(0)[n:], vd.deviceToHostProp(0)[:n][src])


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("kind", ["few cells", "c1", "clump"])
@pytest.mark.parametrize("bc", [(1, 1, 1), (1, 0, 1)])
def test_run_equals_single_steps(pd, dtype, kind, bc):
    x, v, L = _system(kind)
    if bc != (1, 1, 1):
        v = v * [1.0, 0.1, 1.0]
    runs = []
    for parts in ([17], [17], [1] * 17):
        vd, md = _md(pd, x, v, L, bc, dtype)
        E = np.concatenate([md.run(k) for k in parts])
        runs.append((E,) + _by_id(vd))
    assert all(np.array_equal(a, b) for a, b in zip(runs[0], runs[1]))
    assert all(np.array_equal(a, b) for a, b in zip(runs[0], runs[2]))
    assert md.bucket_steps() == 17


def test_large_run_repeats(pd):
    """64,000 particles, every cluster of the GPU and several cells a CTA: what a step's CTAs write is
    there for all of them in the next, so a run repeats bit for bit and equals runs of one step."""
    from openfpm_pdata_b200 import workloads
    x, v, L = workloads.lj_lattice(40, 1.05, 0.05, seed=6)
    runs = []
    for parts in ([60], [60], [1] * 60):
        vd, md = _md(pd, x, v, L, (1, 1, 1), F64)
        runs.append((np.concatenate([md.run(k) for k in parts]),) + _by_id(vd))
    for r in runs[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(runs[0], r))


DT_FLY = 0.002


def _crowding(pd, k, extra=0):
    """Buckets hold 32 records here (0.02 particles a cell on average).  One cell holds 32 particles at
    rest; another flies into it and arrives with step k, leaving after about 60 steps."""
    L = 60.0
    vd = pd.VectorDist(1, np.zeros(3), np.full(3, L), np.ones(3, np.int32), 2.5)
    w = vd.getCellListGPU(2.5).view()
    a = np.array(w.box_lo) + np.array(w.spacing) * 10  # corner of a cell in the middle
    g = np.stack(np.meshgrid(np.arange(4), np.arange(4), np.arange(2), indexing="ij"), -1).reshape(-1, 3)
    rest = a + 0.3 + g * [0.5, 0.5, 0.8]
    rng = np.random.default_rng(7)
    fly = a + [-20.0 * DT_FLY * (k - 0.5), 2.2, 2.2]
    far = rng.uniform(0, L, size=(200, 3))
    far = far[np.abs(far - a).max(1) > 6.0]
    x = np.concatenate([rest, [fly], far])
    v = np.concatenate([np.zeros((32, 3)), [[20.0, 0.0, 0.0]], rng.normal(size=far.shape) * 3])
    return x, v, L


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("k", [1, 2, 4, 5])
def test_bucket_overflow(pd, orc, dtype, k):
    x, v, L = _crowding(pd, k)
    x = x.astype(dtype).astype(F64)
    bc, steps = np.ones(3, np.int32), 12
    t = pd.PD_F64 if dtype == F64 else pd.PD_F32
    runs = []
    for parts in ([steps], [1] * steps):
        vd = pd.VectorDist(len(x), np.zeros(3), np.full(3, L), bc, 2.5, dtype=dtype, props=[(t, 3), (t, 3), (pd.PD_I32, 1)])
        vd.hostToDevicePos(x.astype(dtype))
        vd.hostToDeviceProp(0, v)
        vd.hostToDeviceProp(2, np.arange(len(x)))
        md = pd.MD(vd, 0, 1, dt=DT_FLY, skin=0.0, sigma=0.1, use_cell_list=True)
        E = np.concatenate([md.run(p) for p in parts])
        runs.append((E,) + _by_id(vd))
        assert md.bucket_steps() == k - 1
    xo, vo, Eo = orc.md_lj(x, v, np.zeros(3), np.full(3, L), bc, 2.5, 2.5, 0.0, 1.0, 0.1, DT_FLY, 1.0, steps)
    tol = 1e-9 if dtype == F64 else 1e-4
    np.testing.assert_allclose(runs[0][0][:, :3], Eo[1:, :3], rtol=tol, atol=tol)
    d = runs[0][1] - xo
    assert np.abs(d - L * np.round(d / L)).max() < (1e-9 if dtype == F64 else 1e-3)
    assert np.array_equal(runs[0][1], runs[1][1]) and np.array_equal(runs[0][2], runs[1][2])
    np.testing.assert_allclose(runs[0][0], runs[1][0], rtol=1e-12 if dtype == F64 else 1e-5)
    n = vd.size_local()
    pos = vd.deviceToHostPos()
    img, src, _ = orc.ghost_get(pos[:n], np.zeros(3, dtype), np.full(3, L, dtype), bc, 2.5)
    assert np.array_equal(pos[n:], img)
    assert np.array_equal(vd.deviceToHostProp(0)[n:], vd.deviceToHostProp(0)[:n][src])


def test_returns_to_buckets(pd, orc):
    """The crowd disperses: after some steps on one cluster the buckets are tried again, while it lasts and
    after, in a later run and within one."""
    x, v, L = _crowding(pd, 4)
    bc, steps = np.ones(3, np.int32), 230
    xo, vo, Eo = orc.md_lj(x, v, np.zeros(3), np.full(3, L), bc, 2.5, 2.5, 0.0, 1.0, 0.1, DT_FLY, 1.0, steps)
    for parts in ([steps], [10, 30, 90, 100]):
        vd = pd.VectorDist(len(x), np.zeros(3), np.full(3, L), bc, 2.5, props=[(pd.PD_F64, 3), (pd.PD_F64, 3), (pd.PD_I32, 1)])
        vd.hostToDevicePos(x)
        vd.hostToDeviceProp(0, v)
        vd.hostToDeviceProp(2, np.arange(len(x)))
        md = pd.MD(vd, 0, 1, dt=DT_FLY, skin=0.0, sigma=0.1, use_cell_list=True)
        E = np.concatenate([md.run(p) for p in parts])
        assert 100 < md.bucket_steps() < steps - 32
        np.testing.assert_allclose(E[:, :3], Eo[1:, :3], rtol=1e-9, atol=1e-9)
        d = _by_id(vd)[0] - xo
        assert np.abs(d - L * np.round(d / L)).max() < 1e-9


@pytest.mark.parametrize("dtype", [F32, F64])
def test_one_cluster_from_the_start(pd, orc, dtype):
    """A dense corner of a wide, empty box: two sets of buckets for all its cells would not stay in L2."""
    x, v, _ = _system("clump")
    L, steps = 130.0, 25
    x = x.astype(dtype).astype(F64)
    lo, hi, bc = np.zeros(3), np.full(3, L), np.ones(3, np.int32)
    runs = []
    for parts in ([steps], [1] * steps):
        vd, md = _md(pd, x, v, L, bc, dtype)
        runs.append((np.concatenate([md.run(k) for k in parts]),) + _by_id(vd))
        assert md.bucket_steps() == 0 and md.launch_shape()["cluster_ctas"] in (8, 16)
    assert all(np.array_equal(a, b) for a, b in zip(*runs))
    xo, vo, Eo = orc.md_lj(x, v, lo, hi, bc, 2.5, 2.5, 0.0, 1.0, 1.0, 0.002, 1.0, steps)
    f64 = dtype == F64
    np.testing.assert_allclose(runs[0][0][:, :3], Eo[1:, :3], rtol=1e-9 if f64 else 1e-3, atol=1e-9 if f64 else 1e-2)
    d = runs[0][1] - xo
    assert np.abs(d - L * np.round(d / L)).max() < (1e-9 if f64 else 1e-3)
