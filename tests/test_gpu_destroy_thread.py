"""vt_grid_destroy from a thread that has never made a CUDA call, with the grid's launches still running on
the caller's own stream: the destroy waits for them, so a grid built into the memory given back does not
change their records."""
import threading

import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from test_gpu_parity import assert_hits_equal, hits_from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 64, 96])  # chunk build, graph build, general build
def test_destroy_from_a_fresh_thread_waits_for_the_callers_stream(n):
    import torch
    assert torch.cuda.is_available()
    vt.init(0)
    pal = vt.gen_palette(2)
    vox = vt.gen_cave(n, 2)
    rays = vt.gen_rays_uniform(n, 3, 100000)
    want = po.trace_rays(po.Grid(vox, pal), rays)
    g = vt.Grid.from_u8(vox, pal)
    d_rays = to_dev(torch, rays)
    stream = torch.cuda.Stream()
    bufs = [torch.empty(len(rays) * 16, dtype=torch.uint8, device="cuda") for _ in range(60)]
    torch.cuda.synchronize()
    for b in bufs:
        vt.trace_rays(g, d_rays, len(rays), b, stream)
    other = {}

    def replace():
        try:
            g.destroy()
            other["grid"] = vt.Grid.from_u8(np.zeros_like(vox), pal)
        except Exception as e:
            other["error"] = e

    t = threading.Thread(target=replace)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert "error" not in other, other
    other["grid"].destroy()
    for k in (0, 30, 59):
        assert_hits_equal(hits_from_dev(bufs[k]), want, "launch %d" % k)
