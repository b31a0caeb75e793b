"""Launches too small to fill the chip, which give each warp fewer rays: sizes on both sides of every
step of the rule (2, 4, 8, 16, 32 rays per warp on 152 SMs) and of the ray-buffer form's change, odd
widths and heights, and shadows, against the oracle's records (whole numbers: equality)."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from test_gpu_parity import assert_hits_equal, device_render, device_trace, oracle_camera
from vtrace_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    import torch
    vt.init(0)
    w = workloads.terrain256(n=64)
    g = vt.Grid.from_u8(w["voxels"], w["palette"])
    yield torch, w, g, po.Grid(w["voxels"], w["palette"])
    g.destroy()


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 5803, 5805, 11607, 11609, 23213, 23219, 46427, 46436,
                               196607, 196608])
def test_ray_buffers(scene, n):
    torch, w, g, og = scene
    rays = vt.gen_rays_uniform(64, n, n)
    rays[::7, 3] = 0.0
    hits, _, _ = device_trace(torch, g, rays)
    assert_hits_equal(hits, po.trace_rays(og, rays), "%d rays" % n)


@pytest.mark.parametrize("width,height", [(1, 1), (3, 2), (5, 9), (89, 65), (95, 123), (171, 137), (201, 233), (517, 97)])
@pytest.mark.parametrize("shadows", [False, True])
def test_frames(scene, width, height, shadows):
    torch, w, g, og = scene
    eye, target = workloads.seeded_pose((64, 64, 64), 5, 70.0)
    cam = vt.camera_look_at(eye, target, (0.0, 1.0, 0.0), 60.0, width, height)
    light = workloads.seeded_light(3, shadows=shadows)
    img, _ = device_render(torch, g, cam, light)
    want = po.render(og, oracle_camera(cam), po.make_light(list(light.dir), light.ambient, shadows))
    assert_hits_equal(img, want, "%dx%d" % (width, height))


@pytest.mark.parametrize("sizes", [[(5, 3, 2)], [(40, 30, 1), (33, 17, 3)], [(121, 77, 1), (64, 64, 2)], [(300, 200, 1)]])
def test_batches(scene, sizes):
    torch, w, g, og = scene
    eye, target = workloads.seeded_pose((64, 64, 64), 6, 70.0)
    views, outs = [], []
    for i, (width, height, spp) in enumerate(sizes):
        cam = vt.camera_look_at(eye, target, (0.0, 1.0, 0.0), 60.0, width, height)
        outs.append(torch.full((width * height * spp * 16,), 0xAB, dtype=torch.uint8, device="cuda"))
        views.append(vt.make_view(g, cam, outs[-1], spp, seed=i, view_id=i, light=workloads.seeded_light(4)))
    torch.cuda.synchronize()
    b = vt.Batch(views)
    try:
        saved = []
        for graph in (True, False):
            b.run(torch.cuda.current_stream(), graph=graph)
            torch.cuda.synchronize()
            saved.append([o.cpu().numpy().view(vt.HIT_DTYPE) for o in outs])
            for o in outs:
                o.fill_(0xAB)
        b.stats()  # the counting form walks every iteration, 32 items per warp
        for i, (width, height, spp) in enumerate(sizes):
            want = outs[i].cpu().numpy().view(vt.HIT_DTYPE)
            for got in saved:
                assert_hits_equal(got[i], want, "view %d" % i)
    finally:
        b.destroy()
