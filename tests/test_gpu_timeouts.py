"""A bounded device wait that gave up is reported by the call whose results it spoils, once:
PD_ETIMEOUT, and the next call on the handle runs.  The give-up is made on the host (the error
bit that the kernels set); the wait itself running out is tested in test_gpu_health.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _times_out_once(pd, vd, call):
    call()
    assert pd.lib().pd_selftest_raise_timeout(vd.h) == 0
    with pytest.raises(pd.PdError) as e:
        call()
    assert e.value.code == -5
    call()


@pytest.mark.parametrize("sym", [False, True])
def test_verlet_list(pd, sym):
    rng = np.random.default_rng(1)
    vd = pd.VectorDist(3000, np.zeros(3), np.full(3, 8.0), np.ones(3, np.int32), 1.0)
    vd.hostToDevicePos(rng.uniform(0, 8, size=(3000, 3)))
    vd.ghost_get()
    vl = vd.getVerletSym(1.0) if sym else vd.getVerlet(1.0)
    want = vl.get()
    _times_out_once(pd, vd, lambda: vd.updateVerlet(vl))
    assert all(np.array_equal(a, b) for a, b in zip(vl.get(), want))


@pytest.mark.parametrize("form", ["f64", "f32", "mixed", "global rows", "buckets", "graph"])
@pytest.mark.parametrize("rebuild", [False, True])
def test_md_run(pd, form, rebuild):
    """The run that reports it ends in the middle of a rebuild or between rebuilds; the next ones go on from a
    whole state."""
    from openfpm_pdata_b200 import workloads
    cells = form in ("buckets", "graph")
    x, v, L = workloads.lj_lattice(44 if form == "graph" else 10, 1.1, 0.05, seed=3)
    t = pd.PD_F32 if form in ("f32", "mixed") else pd.PD_F64
    dtype = np.float32 if form == "f32" else np.float64
    vd = pd.VectorDist(len(x), np.zeros(3), np.full(3, L), np.ones(3, np.int32), 2.5 if cells else 2.8, dtype=dtype,
                       props=[(t, 3), (t, 3)])
    vd.hostToDevicePos(x.astype(dtype))
    vd.hostToDeviceProp(0, v)
    skin = 0.0 if cells else (0.002 if rebuild else 0.3)  # 0.002: rebuilt at almost every step
    md = pd.MD(vd, 0, 1, dt=0.001, skin=skin, use_cell_list=cells,
               precision=pd.PREC_MIXED if form == "mixed" else pd.PREC_FP64)
    if form == "global rows":
        md.set_tiles(False)
    E0 = md.run(1)
    _times_out_once(pd, vd, lambda: md.run(2))
    E = md.run(3)
    tot, tot0 = E[:, 0] + E[:, 1], E0[0, 0] + E0[0, 1]
    assert np.abs(tot - tot0).max() < 0.02 * abs(tot0)
    assert np.isfinite(vd.deviceToHostPos()).all()
    if rebuild or cells:
        assert E[:, 3].sum() >= 2
