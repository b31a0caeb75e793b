"""Grid updates where palette index 0 is opaque: a voxel is occupied iff its palette entry's alpha is
nonzero, index 0 included, so cells outside the box keep the occupancy they had and cells past the grid's
faces never get any.  Bricks that no occupied voxel is in (transparent nonzero indices), boxes that end
inside them, partial bricks at the far faces, one-block boxes and larger ones, both element orders; tables,
masks and hits equal those of a fresh build of the updated array."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from test_gpu_parity import assert_hits_equal, device_trace
from test_gpu_update import same_as_fresh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available()
    vt.init(0)
    return t


# one row of one brick; off the brick lattice; the widest box taken in one block is 128 bricks
# (32 x 32 x 64 aligned); 5 x 5 x 6 bricks take the general path, and so does the whole grid
@pytest.mark.parametrize("size", [(3, 1, 1), (13, 9, 11), (16, 16, 16), (32, 32, 64), (40, 40, 45), (67, 50, 83)])
def test_updates_with_an_opaque_index_zero_match_fresh_builds(torch, size):
    dims = (67, 50, 83)
    rng = np.random.default_rng(sum(size))
    pal = vt.gen_palette(4) | np.uint32(0xFF000000)
    pal[9] &= 0x00FFFFFF
    vox = np.full(dims[::-1], 9, np.uint8)  # transparent everywhere: no brick is occupied
    vox[:8, :8, :8] = 0                     # but one, all index 0
    g = vt.Grid.from_u8(vox, pal)
    try:
        lim = [n - s for n, s in zip(dims, size)]
        for step in range(8):
            # against the far faces, in the corner of the occupied brick, then anywhere
            org = lim if step % 4 == 0 else [0, 0, 0] if step == 1 else [int(rng.integers(0, l + 1)) for l in lim]
            box = np.full(size[::-1], 9, np.uint8)
            if step % 3 != 2:
                box[rng.random(size[::-1]) < 0.2] = 5
                box[rng.random(size[::-1]) < 0.2] = 0
            (x, y, z), (w, h, d) = org, size
            vox[z:z + d, y:y + h, x:x + w] = box
            if step % 2:
                g.update(org, np.ascontiguousarray(box.transpose(2, 1, 0)), vt.ORDER_Z_FASTEST)
            else:
                g.update(org, box)
            fresh = vt.Grid.from_u8(vox, pal)
            try:
                same_as_fresh(g, fresh)
            finally:
                fresh.destroy()
        rays = vt.gen_rays_uniform(dims, 7, 20000)
        hits, _, _ = device_trace(torch, g, rays)
        assert_hits_equal(hits, po.trace_rays(po.Grid(vox, pal), rays), "rays after the updates")
    finally:
        g.destroy()
