"""Chunk grids (up to 64 bricks, built in one block) at the limits of the path: one voxel, partial bricks
on every axis, exactly 64 and just more bricks, thin shapes, both formats and element orders, device
input at odd addresses, opaque index 0 and nothing occupied.  Tables, masks and payloads equal the
brute-force layout (whole numbers)."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from test_gpu_build import check_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (16, 16, 16), (13, 7, 22), (32, 32, 32), (33, 32, 32), (31, 29, 30),
                                  (512, 8, 8), (8, 505, 3), (5, 8, 500)])
@pytest.mark.parametrize("density", [0.0, 0.03, 1.0])
def test_chunk_builds_match_the_layout(dims, density):
    import torch
    rng = np.random.default_rng(sum(dims))
    vox = np.where(rng.random(dims[::-1]) < density, rng.integers(1, 256, dims[::-1]), 0).astype(np.uint8)
    pal = vt.gen_palette(2)
    pal[3] &= 0x00FFFFFF
    if density == 0.03:
        pal[0] = 0xFF102030 if dims[0] == 13 else 0  # index 0 opaque: every voxel inside is occupied
    tex = pal[vox]
    d_vox = torch.zeros(vox.size + 3, dtype=torch.uint8, device="cuda")
    d_vox[3:] = torch.from_numpy(vox.reshape(-1)).cuda()
    torch.cuda.synchronize()
    turned = lambda a: np.ascontiguousarray(a.transpose(2, 1, 0))  # noqa: E731
    for make, texels in ((lambda: vt.Grid.from_u8(vox, pal), None),
                         (lambda: vt.Grid.from_rgba8(tex), tex),
                         (lambda: vt.Grid.from_chunk(turned(vox), pal), None),
                         (lambda: vt.Grid.from_chunk(turned(tex)), tex),
                         (lambda: vt.Grid.from_u8_device(d_vox[3:], dims, pal), None)):
        g = make()
        try:
            check_layout(g, vox, pal, texels)
        finally:
            g.destroy()
