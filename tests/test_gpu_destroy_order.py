"""A vector destroyed before its driver (the order of a garbage collector that finds both in
one cycle): the driver leaves the vector's storage alone, so every block of memory keeps one
owner."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


def _system(pd):
    from openfpm_pdata_b200 import workloads
    x, v, L = workloads.lj_lattice(10, 1.1, 0.05, seed=9)
    vd = pd.VectorDist(len(x), np.zeros(3), np.full(3, L), np.ones(3, np.int32), 2.8,
                       props=[(pd.PD_F64, 3), (pd.PD_F64, 3)])
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, v)
    return vd, pd.MD(vd, 0, 1, dt=0.005, skin=0.3), len(x)


def test_vector_destroyed_first(pd):
    want = _system(pd)[1].run(40)
    for _ in range(4):
        vd, md, n = _system(pd)
        md.run(3)
        pd.lib().pd_destroy(vd.h)
        vd.h = None
        pd.lib().pd_md_destroy(md.h)
        md.h = None
    gc.collect()
    some = [_system(pd) for _ in range(6)]
    spans = []
    for vd, _, n in some:
        w = vd.toKernel()
        spans += [(w.pos, 32 * n)] + [(w.prop[p], 24 * n) for p in range(2)]
    spans.sort()
    assert all(a + m <= b for (a, m), (b, _) in zip(spans, spans[1:]))
    for _, md, _ in some:
        assert np.array_equal(md.run(40), want)
