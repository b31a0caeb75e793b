"""Which form a ray buffer takes: the built-in tuning leaves small buffers to one thread per ray, an
installed one is taken as it is at every size.  Seen from the graph nodes of a captured call: the
persistent form clears its work counter first.  The records are the oracle's either way."""
import ctypes

import numpy as np
import pytest

import vtrace_gb300 as vt
from vtrace_gb300 import autotune
from oracle import pyoracle as po
from test_gpu_parity import assert_hits_equal, hits_from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    import torch
    assert torch.cuda.is_available()
    vt.init(0)
    vox, pal = vt.gen_cave(40, 2), vt.gen_palette(2)
    g = vt.Grid.from_u8(vox, pal)
    yield torch, g, po.Grid(vox, pal)
    g.destroy()


def captured_nodes(torch, fn):
    """Nodes of the graph that fn(stream) records."""
    cu = ctypes.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    handle, graph, n = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert cu.cuStreamBeginCapture_v2(handle, 1) == 0  # thread-local mode
    try:
        fn(stream)
    finally:
        rc = cu.cuStreamEndCapture(handle, ctypes.byref(graph))
    assert rc == 0
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    assert cu.cuGraphDestroy(graph) == 0
    return n.value


def test_installed_tuning_holds_at_every_size(scene):
    torch, g, og = scene
    saved = vt.get_tuning(vt.KERNEL_TRACE_RAYS)
    small, large = 4099, 196608
    rays = vt.gen_rays_uniform(40, 3, large)
    d_rays = to_dev(torch, rays)
    d_hits = torch.empty(large * 16, dtype=torch.uint8, device="cuda")
    want = po.trace_rays(og, rays)

    def nodes(n):
        return captured_nodes(torch, lambda s: vt.trace_rays(g, d_rays, n, d_hits, s))

    try:
        # as the library starts
        assert (nodes(small), nodes(large - 1), nodes(large)) == (1, 1, 2)
        for c in autotune.rays_candidates():
            if {k: int(v) for k, v in c.items()} == {k: int(v) for k, v in saved.items()}:
                continue
            autotune.install(vt.KERNEL_TRACE_RAYS, c)
            form = 2 if c["persistent"] else 1
            assert (nodes(small), nodes(large)) == (form, form), c
            for n in (1, small):
                d_hits.zero_()
                vt.trace_rays(g, d_rays, n, d_hits)
                torch.cuda.synchronize()
                assert_hits_equal(hits_from_dev(d_hits)[:n], want[:n], str(c))
        # putting the built-in tuning back puts its rule back
        vt.set_tuning(vt.KERNEL_TRACE_RAYS, **saved)
        assert (nodes(small), nodes(large)) == (1, 2)
    finally:
        vt.set_tuning(vt.KERNEL_TRACE_RAYS, **saved)
