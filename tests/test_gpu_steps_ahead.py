"""Steps enqueued ahead of their rebuild decision: a run equals runs of one step bit for
bit (each of those decides before it enqueues), for lists that are rebuilt at almost every
step, every few steps and never within the run, for every driver."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _lj(pd, form, skin, n_side, T):
    from openfpm_pdata_b200 import workloads
    x, v, L = workloads.lj_lattice(n_side, 1.1, 0.05, seed=3, temperature=T)
    dt = F32 if form == "f32" else F64
    t = pd.PD_F64 if form == "f64" else pd.PD_F32
    vd = pd.VectorDist(x.shape[0], np.zeros(3), np.full(3, L), np.ones(3, np.int32), 2.5 + skin, dtype=dt,
                       props=[(t, 3), (t, 3), (pd.PD_I32, 1)])
    vd.hostToDevicePos(x.astype(dt))
    vd.hostToDeviceProp(0, v)
    vd.hostToDeviceProp(2, np.arange(x.shape[0]))
    return vd, pd.MD(vd, 0, 1, dt=0.005, skin=skin,
                     precision=pd.PREC_MIXED if form == "mixed" else pd.PREC_FP64)


def _state(vd, ids, props):
    i = vd.deviceToHostProp(ids, with_ghost=False)
    out = []
    for a in [vd.deviceToHostPos(with_ghost=False)] + [vd.deviceToHostProp(p, with_ghost=False) for p in props]:
        b = np.empty_like(a)
        b[i] = a
        out.append(b)
    return out


@pytest.mark.parametrize("form", ["f64", "f32", "mixed"])
@pytest.mark.parametrize("skin,n_side,T", [(0.01, 9, 1.0), (0.12, 9, 1.0), (0.3, 13, 3.0), (1.0, 9, 0.2)])
def test_lj_run_equals_single_steps(pd, form, skin, n_side, T):
    steps = 27
    a, ma = _lj(pd, form, skin, n_side, T)
    b, mb = _lj(pd, form, skin, n_side, T)
    Ea = np.concatenate([ma.run(20), ma.run(steps - 20)])
    Eb = np.concatenate([mb.run(1) for _ in range(steps)])
    assert np.array_equal(Ea, Eb)
    for p, q in zip(_state(a, 2, [0]), _state(b, 2, [0])):
        assert np.array_equal(p, q)
    assert ma.stats() == mb.stats()


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("skin", [0.002, 0.3])
def test_sph_run_equals_single_steps(pd, dtype, skin):
    from openfpm_pdata_b200 import workloads
    dp, steps = 1.0 / 20, 21
    x, typ, m, lo, hi = workloads.sph_dam(dp)
    t = pd.PD_F32 if dtype == F32 else pd.PD_F64
    rng = np.random.default_rng(1)
    v = np.where(typ[:, None] == 0, rng.normal(0, 0.5, size=x.shape), 0.0)
    runs = []
    for one in (False, True):
        vd = pd.VectorDist(x.shape[0], lo, hi, np.zeros(3, np.int32), 0.0, dtype=dtype,
                           props=[(t, 3), (t, 3), (t, 1), (t, 1), (pd.PD_I32, 1), (pd.PD_I32, 1)])
        vd.hostToDevicePos(x.astype(dtype))
        vd.hostToDeviceProp(0, v)
        vd.hostToDeviceProp(2, np.full(x.shape[0], 1000.0))
        vd.hostToDeviceProp(4, typ)
        vd.hostToDeviceProp(5, np.arange(x.shape[0]))
        s = pd.SPH(vd, 0, 1, 2, 3, 4, 1.3 * dp, m, 20.0, 1000.0, 0.1, -9.81, 1e-4, skin=skin * dp)
        E = np.concatenate([s.run(1) for _ in range(steps)]) if one else s.run(steps)
        runs.append((E, _state(vd, 5, [0, 2]), s.stats()))
    assert np.array_equal(runs[0][0], runs[1][0])
    for p, q in zip(runs[0][1], runs[1][1]):
        assert np.array_equal(p, q)
    assert runs[0][2] == runs[1][2]
