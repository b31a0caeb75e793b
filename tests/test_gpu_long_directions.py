"""Rays whose direction is so long that its squares overflow (about 1.8e19 and more): side distances are
infinite, all axes with a component step together, and at the far face of a grid one voxel wide the first
side is -inf.  Every form of the traversal gives the oracle's records, in dense bricks, sparse ones and
empty space, for directions along an axis, in a plane and in space.  (t can be 0 * inf: one NaN is as good as
another, the two machines' differ in their bits.)"""
import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from test_gpu_parity import assert_hits_equal as records_equal, device_trace, hits_from_dev

pytestmark = pytest.mark.gpu


def assert_hits_equal(got, want, what):
    got, want = got.copy(), want.copy()
    for h in (got, want):
        h["t"][np.isnan(h["t"])] = np.nan
    records_equal(got, want, what)


def overflowing_rays(dims, seed, n):
    rng = np.random.default_rng(seed)
    size = np.array(dims, np.float64)
    o = rng.random((n, 3)) * size
    o[::5] = np.floor(o[::5])                                     # on voxel faces: 0 * inf
    kind = rng.integers(0, 3, n)
    face = np.where(rng.random((n, 3)) < 0.5, 0.0, size)
    o = np.where((np.arange(3) == kind[:, None]) & (np.arange(n) % 3 == 0)[:, None], face, o)
    o = o.astype(np.float32)
    past = rng.random((n, 3)) < 0.15                              # one step past the face, either way
    o = np.where(past, np.nextafter(o, np.where(o > size / 2, np.inf, -np.inf).astype(np.float32)), o)
    d = rng.normal(size=(n, 3))
    d[rng.random((n, 3)) < 0.35] = 0.0
    d *= 10.0 ** rng.uniform(18, 38, (n, 1))
    return np.concatenate([o, np.clip(d, -3.3e38, 3.3e38)], 1).astype(np.float32)


@pytest.mark.parametrize("dims", [(1, 13, 13), (13, 1, 2), (5, 3, 1), (1, 1, 1), (40, 24, 33), (203, 9, 64)])
@pytest.mark.parametrize("fill", [0.0, 0.002, 0.4])
def test_overflowing_directions_give_the_oracles_records(dims, fill):
    import torch
    assert torch.cuda.is_available()
    vt.init(0)
    rng = np.random.default_rng(sum(dims))
    vox = np.where(rng.random(dims[::-1]) < fill, 3, 0).astype(np.uint8)
    vox[0, 0, 0] = 2  # the first brick is occupied
    pal = vt.gen_palette(1)
    rays = overflowing_rays(dims, 5, 4000)
    # one voxel wide: at the face, a last place past it, along the axis alone
    for a in range(3):
        edge = np.tile(np.array([0.5, 0.5, 0.5, 0, 0, 0], np.float32), (4, 1))
        edge[:, :3] = np.array(dims) * 0.5
        edge[:, a] = [dims[a], np.nextafter(np.float32(dims[a]), np.float32(np.inf)), 0, -1e-45]
        edge[:, 3 + a] = [3e38, 3e38, -3e38, -3e38]
        rays = np.concatenate([rays, edge])
    want = po.trace_rays(po.Grid(vox, pal), rays)
    g = vt.Grid.from_u8(vox, pal)
    saved = vt.get_tuning(vt.KERNEL_TRACE_RAYS)
    try:
        hits, d_rays, d_hits = device_trace(torch, g, rays)
        assert_hits_equal(hits, want, "one thread per ray")
        vt.set_tuning(vt.KERNEL_TRACE_RAYS, 4, 0, True)
        d_hits.zero_()
        vt.trace_rays(g, d_rays, len(rays), d_hits)
        torch.cuda.synchronize()
        assert_hits_equal(hits_from_dev(d_hits), want, "resident warps")
        d_hits.zero_()
        vt.trace_rays_stats(g, d_rays, len(rays), d_hits)
        assert_hits_equal(hits_from_dev(d_hits), want, "counting form")
    finally:
        vt.set_tuning(vt.KERNEL_TRACE_RAYS, **saved)
        g.destroy()
