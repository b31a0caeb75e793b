"""The path tracer's ray queues where they change course: no bounce, the last vertex's sun rays alone,
one pixel, and queues longer than one round of the grid-stride shading, against the oracle's estimator
(float radiance bit for bit, the same number of rays)."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from vtrace_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,spp,bounces,sun", [
    (33, 17, 2, 0, True), (33, 17, 2, 0, False), (57, 31, 1, 1, True), (57, 31, 1, 1, False),
    (1, 1, 3, 2, True), (8, 4, 17, 2, True), (900, 700, 1, 2, True),
])
def test_queues_match_the_oracle(width, height, spp, bounces, sun):
    w = workloads.terrain256(n=64, width=width, height=height)
    p = vt.make_path_params(spp=spp, max_bounces=bounces, seed=4, **({} if sun else {"sun": (0.0, 0.0, 0.0)}))
    g = vt.Grid.from_u8(w["voxels"], w["palette"])
    try:
        got, rays = vt.path_trace_host(g, w["camera"], p)
        want, want_rays = po.path_trace(
            po.Grid(w["voxels"], w["palette"]), po.make_camera(w["camera"].as_dict()),
            po.make_path_params(p.spp, p.max_bounces, p.seed, list(p.sky), list(p.sun_dir), list(p.sun)))
        np.testing.assert_array_equal(got, want)
        assert rays == want_rays
    finally:
        g.destroy()
