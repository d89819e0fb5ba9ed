"""Kernels that work in tiles, at the edges of the tiles and where the prefix sums over them
change their form: the scan of a cell list's counts, ghost images, compaction, index
selection, sorted domain slots, multi-column reorders, and the device-array copies, all exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F32, F64 = np.float32, np.float64


@pytest.fixture(scope="module")
def pd():
    from openfpm_pdata_b200 import pd as _pd
    _pd.lib()
    return _pd


@pytest.mark.parametrize("gs", [(3, 4, 5), (11, 12, 31), (13, 15, 21), (16, 16, 16), (15, 17, 257), (32, 32, 64),
                                (45, 17, 257), (64, 64, 48), (128, 128, 257), (31, 601, 1801), (256, 256, 512)])
def test_cell_starts(pd, gs):
    """Cell starts are the exclusive scan of the counts: cells + 1 elements, 4093, 4096 and 4097
    among them (one tile, two), 65536 and 65537, 196606 and 196609 (the last tiles that one launch
    scans), 33554432 and 33554433 (the last that each add up the ones before).  Twice in a row."""
    rng = np.random.default_rng(sum(gs))
    L = np.array(gs) - 2.5
    n = 20011
    x = rng.random((n, 3)) * L
    x[: n // 3] = L - rng.random((n // 3, 3)) * np.minimum(L, 2.0)  # many in the last cells
    vd = pd.VectorDist(n, np.zeros(3), L, np.zeros(3, np.int32), 0.0)
    vd.hostToDevicePos(x)
    cl = vd.getCellListGPU(1.0)
    v = cl.view()
    assert tuple(v.gs) == gs
    c = np.floor((x - np.array(v.box_lo)) / np.array(v.spacing)).astype(np.int64) + v.pad
    cell = c[:, 0] + gs[0] * (c[:, 1] + gs[1] * c[:, 2])
    want = np.concatenate([[0], np.cumsum(np.bincount(cell, minlength=v.ncells))])
    for _ in range(2):
        vd.updateCellListGPU(cl)
        cs, so = cl.get()
        assert np.array_equal(cs, want)
        assert np.array_equal(so, np.argsort(cell, kind="stable"))


def test_many_tiles(pd, orc):
    """More tiles than add up their predecessors: ghost images (1,024 particles a tile), index
    selection and removal (4,096)."""
    import torch
    n, g = 8400001, 0.01
    lo, hi, bc = np.zeros(3), np.ones(3), np.ones(3, np.int32)
    x = np.random.default_rng(8).random((n, 3), dtype=F32)
    vd = pd.VectorDist(n, lo, hi, bc, g, dtype=F32)
    vd.hostToDevicePos(x)
    vd.ghost_get()
    img, src, _ = orc.ghost_get(x, lo.astype(F32), hi.astype(F32), bc, g)
    assert np.array_equal(vd.ghost_records()[0], src)
    assert np.array_equal(vd.deviceToHostPos()[n:], img)
    del vd
    n = 8193 * 4096 + 5
    vd = pd.VectorDist(n, lo, hi, bc, g, dtype=F32, props=[(pd.PD_I32, 1)])
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand((n, 3), device="cuda", generator=gen)
    mark = (torch.rand(n, device="cuda", generator=gen) < 0.2).int()
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, mark)
    assert torch.equal(vd.get_indexes_by_type(0, 1, device=True).long(), mark.nonzero()[:, 0])
    vd.remove_marked(0)
    assert torch.equal(vd.deviceToHostPos(device=True), x[mark == 0])


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n,corner", [(1, True), (1023, False), (1024, False), (1025, True), (40000, False),
                                      (20001, True)])
def test_ghost_images(pd, orc, dtype, n, corner):
    """Images, sources and shifts of several calls; with every particle in one corner (seven
    images each) the first call finds far more images than it made room for."""
    rng = np.random.default_rng(n)
    L, g = 4.0, 0.25
    lo, hi, bc = np.zeros(3), np.full(3, L), np.ones(3, np.int32)
    vd = pd.VectorDist(n, lo, hi, bc, g, dtype=dtype, props=[(pd.PD_I32, 1), (pd.PD_F64, 2)])
    a = np.arange(n, dtype=np.int32)
    b = rng.normal(size=(n, 2))
    for rep in range(3):
        x = rng.uniform(0, 0.2 if corner and rep != 1 else L, size=(n, 3)).astype(dtype)
        x = orc.wrap(x, lo.astype(dtype), hi.astype(dtype), bc)
        vd.map()
        vd.hostToDevicePos(x)
        vd.hostToDeviceProp(0, a)
        vd.hostToDeviceProp(1, b)
        vd.ghost_get()
        img, src, shf = orc.ghost_get(x, lo.astype(dtype), hi.astype(dtype), bc, g)
        s, h = vd.ghost_records()
        assert np.array_equal(s, src) and np.array_equal(h, shf)
        assert np.array_equal(vd.deviceToHostPos()[n:], img)
        assert np.array_equal(vd.deviceToHostProp(0)[n:], a[src])
        assert np.array_equal(vd.deviceToHostProp(1)[n:], b[src])


def test_ghost_boxes_after_user_boxes(pd, orc):
    """The domain's boxes, uploaded once, come back after a call with other boxes."""
    rng = np.random.default_rng(3)
    lo, hi, bc = np.zeros(3), np.ones(3), np.ones(3, np.int32)
    x = rng.random((5000, 3))
    vd = pd.VectorDist(5000, lo, hi, bc, 0.1)
    vd.hostToDevicePos(x)
    vd.ghost_get()
    _, src, _ = orc.ghost_get(x, lo, hi, bc, 0.1)
    vd.ghost_count_boxes([[0, 0, 0]], [[0.5, 0.5, 0.5]], [0])
    vd.ghost_get()
    assert np.array_equal(vd.ghost_records()[0], src)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 70001])
@pytest.mark.parametrize("frac", [0.0, 0.3, 1.0])
def test_remove_and_indexes(pd, orc, n, frac):
    rng = np.random.default_rng(n)
    lo, hi, bc = np.zeros(3), np.ones(3), np.ones(3, np.int32)
    # 2 + 1 + 30 columns: more than one launch takes
    vd = pd.VectorDist(n, lo, hi, bc, 0.1, props=[(pd.PD_I32, 1), (pd.PD_F32, 30)])
    x, p = rng.random((n, 3)), rng.normal(size=(n, 30)).astype(F32)
    mark = (rng.random(n) < frac).astype(np.int32)
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, mark)
    vd.hostToDeviceProp(1, p)
    want = np.nonzero(mark == 1)[0]
    assert np.array_equal(vd.get_indexes_by_type(0, 1), want)
    assert np.array_equal(vd.get_indexes_by_type(0, 1, device=True).cpu().numpy(), want)
    assert np.array_equal(vd.get_indexes_by_type(0, 1, end=n // 2), want[want < n // 2])
    vd.remove_marked(0)
    keep = mark == 0
    assert vd.size_local() == keep.sum()
    assert np.array_equal(vd.deviceToHostPos(), x[keep])
    assert np.array_equal(vd.deviceToHostProp(1), p[keep])
    assert np.array_equal(vd.gid(), np.nonzero(keep)[0])


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n", [1, 2047, 2049, 30011])
def test_reorder_many_columns(pd, dtype, n):
    """22 columns of 4 and 8 bytes there and back, with ghosts; the sorted domain slots."""
    rng = np.random.default_rng(n)
    vd = pd.VectorDist(n, np.zeros(3), np.ones(3), np.ones(3, np.int32), 0.1, dtype=dtype,
                       props=[(pd.PD_F64, 13), (pd.PD_F32, 5), (pd.PD_I64, 2)])
    x = rng.random((n, 3)).astype(dtype)
    vals = [rng.normal(size=(n, 13)), rng.normal(size=(n, 5)).astype(F32), rng.integers(-9, 9, size=(n, 2))]
    vd.hostToDevicePos(x)
    for p, a in enumerate(vals):
        vd.hostToDeviceProp(p, a)
    vd.ghost_get()
    before = [vd.deviceToHostPos(), vd.gid()] + [vd.deviceToHostProp(p) for p in range(3)]
    cl = vd.getCellListGPU(0.1, opt=pd.CL_NON_SYMMETRIC | pd.CL_GPU_REORDER)
    vd.updateCellListGPU(cl)
    _, so = cl.get()
    after = [vd.deviceToHostPos(), vd.gid()] + [vd.deviceToHostProp(p) for p in range(3)]
    for a, b in zip(before, after):
        assert np.array_equal(a[so], b)
    import torch
    view = cl.view()
    dom = torch.empty(n, dtype=torch.int32, device="cuda")
    import ctypes
    ctypes.CDLL("libcudart.so.12").cudaMemcpy(ctypes.c_void_p(dom.data_ptr()), ctypes.c_void_p(view.dom_sort_ids),
                                              ctypes.c_size_t(4 * n), ctypes.c_int(3))
    assert np.array_equal(dom.cpu().numpy(), np.nonzero(so < n)[0])
    vd.restoreOrder(cl)
    for a, b in zip(before, [vd.deviceToHostPos(), vd.gid()] + [vd.deviceToHostProp(p) for p in range(3)]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("n", [1, 1001])
def test_device_arrays(pd, dtype, n):
    """Device tensors in and out, whole, sliced, at offsets, strided and one element off."""
    import torch
    t = torch.float32 if dtype == F32 else torch.float64
    pt = pd.PD_F32 if dtype == F32 else pd.PD_F64
    vd = pd.VectorDist(n, np.zeros(3), np.ones(3), np.ones(3, np.int32), 0.1, dtype=dtype,
                       props=[(pt, 3), (pd.PD_I32, 1), (pd.PD_I64, 2)])
    g = torch.Generator(device="cuda").manual_seed(1)
    flat = torch.rand(3 * n + 1, device="cuda", dtype=t, generator=g)
    x = flat[1:].reshape(n, 3)  # starts one element past the allocation
    wide = torch.rand((n, 6), device="cuda", dtype=t, generator=g)
    v = wide[:, ::2]
    i32 = torch.arange(n, device="cuda", dtype=torch.int32)
    i64 = torch.arange(2 * n, device="cuda").reshape(n, 2) - n
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, v)
    vd.hostToDeviceProp(1, i32)
    vd.hostToDeviceProp(2, i64)
    assert torch.equal(vd.deviceToHostPos(device=True), x)
    assert torch.equal(vd.deviceToHostProp(0, device=True), v)
    assert torch.equal(vd.deviceToHostProp(1, device=True), i32)
    assert torch.equal(vd.deviceToHostProp(2, device=True), i64)
    assert np.array_equal(vd.deviceToHostPos(), x.cpu().numpy())
    assert np.array_equal(vd.deviceToHostProp(0), v.cpu().numpy())
    if n > 1:
        vd.hostToDeviceProp(0, v[:7] * 2, offset=3)
        assert torch.equal(vd.deviceToHostProp(0, offset=2, count=9, device=True),
                           torch.cat([v[2:3], v[:7] * 2, v[10:11]]))
        assert torch.equal(vd.deviceToHostPos(offset=5, count=11, device=True), x[5:16])


def test_positions_complete_on_return(pd):
    """deviceToHostPos(device=True) returns when the positions are there: another stream may
    read the tensor at once, although the device was busy at the call."""
    import torch
    n = 5000
    x = np.random.default_rng(2).random((n, 3))
    vd = pd.VectorDist(n, np.zeros(3), np.ones(3), np.ones(3, np.int32), 0.1)
    vd.hostToDevicePos(x)
    side = torch.cuda.Stream()
    torch.cuda._sleep(1 << 27)  # about 70 ms of the default stream
    t = vd.deviceToHostPos(device=True)
    assert torch.cuda.default_stream().query()
    with torch.cuda.stream(side):
        got = t.cpu()
    assert np.array_equal(got.numpy(), x)


def test_reorder_scratch(pd):
    """A reorder of a large vector takes scratch for its largest column, not for all of them."""
    import ctypes
    import torch
    n = 8000003

    def free():
        torch.cuda.synchronize()
        f = ctypes.c_long(0)
        assert pd.lib().pd_device_info(None, ctypes.byref(f), None) == 0
        return f.value

    vd = pd.VectorDist(n, np.zeros(3), np.ones(3), np.zeros(3, np.int32), 0.0, props=[(pd.PD_F64, 7), (pd.PD_F32, 2)])
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand((n, 3), device="cuda", dtype=torch.float64, generator=gen)
    p = torch.rand((n, 7), device="cuda", dtype=torch.float64, generator=gen)
    vd.hostToDevicePos(x)
    vd.hostToDeviceProp(0, p)
    cl = vd.getCellListGPU(0.01, opt=pd.CL_NON_SYMMETRIC)
    vd.updateCellListGPU(cl)  # the sort's own buffers
    cr = vd.getCellListGPU(0.01, opt=pd.CL_NON_SYMMETRIC | pd.CL_GPU_REORDER)
    pd.lib().pd_empty_cache()
    before = free()
    vd.updateCellListGPU(cr)
    sort = 5 * 4 * n + 3 * 4 * cr.view().ncells
    assert before - free() < sort + 32 * n + (64 << 20)
    so = torch.from_numpy(cr.get()[1].astype(np.int64)).cuda()
    assert torch.equal(vd.deviceToHostPos(device=True), x[so])
    assert torch.equal(vd.deviceToHostProp(0, device=True), p[so])
    vd.restoreOrder(cr)
    assert torch.equal(vd.deviceToHostPos(device=True), x)
    assert torch.equal(vd.deviceToHostProp(0, device=True), p)


def test_ghost_get_near_the_memory_limit(pd):
    """The room made for images before the first count is an estimate: where memory does not
    suffice for it, particles that have no image need none."""
    import torch
    n = 400000
    lo, hi, bc = np.zeros(3), np.ones(3), np.ones(3, np.int32)
    vd = pd.VectorDist(n, lo, hi, bc, 0.49, props=[(pd.PD_F64, 64), (pd.PD_F64, 64)])
    x = 0.5 + (np.random.default_rng(4).random((n, 3)) - 0.5) * 0.01
    x[:5] = 0.1
    vd.hostToDevicePos(x)
    pd.lib().pd_empty_cache()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")  # 4.5 GB were wanted
    try:
        vd.ghost_get([])
        vd.ghost_get([])
    finally:
        del block
        torch.cuda.empty_cache()
    assert vd.size_local_with_ghost() == n + 5 * 7
    got = vd.deviceToHostPos()
    assert np.array_equal(got[:n], x)
    assert np.array_equal(np.unique(got[n:].round(6)), [0.1, 1.1])
