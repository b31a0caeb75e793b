"""Calls that take voxels from host memory see what earlier work on the library's stream wrote there: a
copy into page-locked memory queued behind device work, then a build or an update from that memory
without a wait in between.  The sizes take the one-block chunk build, the graph build, the general
build, the one-block update and the general update."""
import ctypes

import numpy as np
import pytest

import vtrace_gb300 as vt
from test_gpu_update import same_as_fresh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available()
    vt.init(0)
    return t


@pytest.fixture
def queued(torch):
    """queued(array): page-locked zeros that a copy of `array`, queued on the library's stream behind
    some milliseconds of work, is about to fill."""
    stream = torch.cuda.ExternalStream(vt.lib().vt_get_stream())
    busy = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")

    def put(array):
        src = torch.from_numpy(np.ascontiguousarray(array).reshape(-1)).cuda()
        dst = torch.zeros(src.numel(), dtype=torch.uint8, pin_memory=True)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(40):
                busy.fill_(1)
            dst.copy_(src, non_blocking=True)
        src.record_stream(stream)
        return dst

    yield put
    torch.cuda.synchronize()


@pytest.mark.parametrize("n", [16, 48, 96])
def test_device_addresses_are_taken(torch, n):
    pal = vt.gen_palette(3)
    vox = vt.gen_shapes(n, 5, count=12, rmin=2, rmax=n / 4)
    dev = torch.from_numpy(vox.reshape(-1)).cuda()
    devz = torch.from_numpy(np.ascontiguousarray(vox.transpose(2, 1, 0)).reshape(-1)).cuda()
    empty = vt.Grid.from_u8(np.zeros_like(vox), pal)
    vt.check(vt.lib().vt_grid_update(empty.id, dev.data_ptr(), vt.ORDER_X_FASTEST, 0, 0, 0, n, n, n))
    made = [empty] + [vt.Grid(vt.check(vt.lib().vt_grid_create(d.data_ptr(), vt.PAYLOAD_U8, order, pal.ctypes.data, n, n, n)))
                      for d, order in ((dev, vt.ORDER_X_FASTEST), (devz, vt.ORDER_Z_FASTEST))]
    fresh = vt.Grid.from_u8(vox, pal)
    try:
        for g in made:
            same_as_fresh(g, fresh)
    finally:
        for g in made + [fresh]:
            g.destroy()


@pytest.mark.parametrize("order", [vt.ORDER_X_FASTEST, vt.ORDER_Z_FASTEST])
@pytest.mark.parametrize("n", [16, 48, 96])
def test_build_sees_the_stream_ordered_copy(torch, queued, n, order):
    pal = vt.gen_palette(3)
    vox = vt.gen_shapes(n, 5, count=12, rmin=2, rmax=n / 4)
    host = queued(vox if order == vt.ORDER_X_FASTEST else vox.transpose(2, 1, 0))
    g = vt.Grid(vt.check(vt.lib().vt_grid_create(host.data_ptr(), vt.PAYLOAD_U8, order, pal.ctypes.data, n, n, n)))
    fresh = vt.Grid.from_u8(vox, pal)
    try:
        assert fresh.info()["voxels_occupied"] > 0
        same_as_fresh(g, fresh)
    finally:
        g.destroy()
        fresh.destroy()


@pytest.mark.parametrize("size", [16, 48])
def test_update_sees_the_stream_ordered_copy(torch, queued, size):
    pal = vt.gen_palette(3)
    vox = np.zeros((64, 64, 64), np.uint8)
    g = vt.Grid.from_u8(vox, pal)
    box = vt.gen_shapes(size, 6, count=12, rmin=2, rmax=size / 4)
    vox[8:8 + size, 8:8 + size, 8:8 + size] = box
    host = queued(box)
    vt.check(vt.lib().vt_grid_update(g.id, ctypes.c_void_p(host.data_ptr()), vt.ORDER_X_FASTEST, 8, 8, 8, size, size, size))
    fresh = vt.Grid.from_u8(vox, pal)
    try:
        same_as_fresh(g, fresh)
    finally:
        g.destroy()
        fresh.destroy()
