"""The service's traces keep each sample's colour alone: its images equal the per-channel averages of
the full records that a view batch writes for the same views, in the tile form and the refilled one."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from vtrace_gb300 import workloads
from test_gpu_serve import oracle_image, pinned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refill", [32, 8])
@pytest.mark.parametrize("size,spp", [((1, 1), 1), ((9, 5), 3), ((131, 67), 2), ((200, 33), 5)])
def test_colours_match_the_oracle(refill, size, spp):
    torch = pytest.importorskip("torch")
    vt.init(0)
    scenes, views = workloads.multiview(n_scenes=2, n_views=4, sizes=(40, 64), min_px=200, max_px=400)
    svc = vt.Service(max_inflight=2, refill_min=refill)
    try:
        sids = [svc.add_scene(s["voxels"], s["palette"]) for s in scenes]
        out = []
        for v in views:
            v["camera"].width, v["camera"].height = size
            v["spp"] = spp
            host = pinned(torch, v["camera"])
            out.append((svc.submit(sids[v["scene"]], v["camera"], host, spp, v["seed"],
                                   v["view_id"], v["light"]), host))
        for v, (req, host) in zip(views, out):
            svc.wait(req)
            want = oracle_image(scenes[v["scene"]], v)
            assert np.array_equal(host.numpy().reshape(want.shape), want)
    finally:
        svc.stop()
