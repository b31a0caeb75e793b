"""Small grid updates (taken in one block): brick counts at the limits of the path (one brick, 128 and
more), boxes off the brick lattice and at the grid's partial bricks, both element orders and formats,
slots freed and handed out in the same call, and slot arrays that have to grow.  Tables, masks and
occupied voxels equal those of fresh builds, and slot numbers the free list's order (whole numbers)."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from test_gpu_update import same_as_fresh

pytestmark = pytest.mark.gpu


def payload_by_brick(g):
    """Voxels of the occupied bricks, in brick order, where they are occupied (0 elsewhere): a brick
    with no occupied voxel has no slot, so what transparent voxels it was given is not kept."""
    d, m = g.bricks()
    full = np.nonzero((d & 0x80000000) == 0)[0]
    bits = ((m[d[full]][:, :, None] >> np.arange(64, dtype=np.uint64)) & np.uint64(1)).astype(bool)
    p = g.payload()[d[full]]
    bits = bits.reshape(p.shape[:4])
    return full, np.where(bits[..., None] if p.ndim == 5 else bits, p, 0)


@pytest.mark.parametrize("rgba", [False, True])
@pytest.mark.parametrize("dims", [(67, 50, 83), (136, 130, 40)])
def test_small_updates_match_fresh_builds(dims, rgba):
    rng = np.random.default_rng(sum(dims) + rgba)
    pal = vt.gen_palette(6)
    pal[9] &= 0x00FFFFFF  # stored, not occupied
    vox = np.zeros(dims[::-1], np.uint8)
    vox[:20, :20, :20] = 3
    make = (lambda v: vt.Grid.from_rgba8(pal[v])) if rgba else (lambda v: vt.Grid.from_u8(v, pal))
    g = make(vox)
    # 1 brick; 2 x 2 x 2; 27 off the lattice; 4 x 4 x 8 = 128; 5 x 5 x 6 = 150 (general path)
    sizes = [(8, 8, 8), (16, 16, 16), (16, 16, 16), (1, 1, 1), (32, 32, 64), (40, 40, 45), (17, 3, 20)]
    aligned = [True, True, False, False, True, True, False]
    try:
        for step in range(21):
            i = step % len(sizes)
            size = [min(s, n) for s, n in zip(sizes[i], dims)]
            lim = [n - s for n, s in zip(dims, size)]
            org = [int(rng.integers(0, l // 8 + 1)) * 8 if aligned[i] else int(rng.integers(0, l + 1)) for l in lim]
            if step % 4 == 1:
                org = lim  # against the far faces
            box = np.where(rng.random(size[::-1]) < (0.0 if step % 3 == 2 else 0.02), 5, 0).astype(np.uint8)
            box[rng.random(size[::-1]) < 0.01] = 9
            (x, y, z), (w, h, d) = org, size
            vox[z:z + d, y:y + h, x:x + w] = box
            data = pal[box] if rgba else box
            if step % 2:
                g.update(org, np.ascontiguousarray(data.transpose(2, 1, 0)), vt.ORDER_Z_FASTEST)
            else:
                g.update(org, data)
            fresh = make(vox)
            try:
                same_as_fresh(g, fresh)
                a, b = payload_by_brick(g), payload_by_brick(fresh)
                np.testing.assert_array_equal(a[0], b[0])
                np.testing.assert_array_equal(a[1], b[1])
            finally:
                fresh.destroy()
    finally:
        g.destroy()


def test_slots_are_handed_out_in_brick_order():
    # four bricks emptied and four filled by one box: the freed slots come back last freed first, then
    # the older free slots, then new ones
    pal = vt.gen_palette(2)
    vox = np.zeros((8, 8, 128), np.uint8)
    vox[..., 8:72] = 1  # bricks 1..8: slots 0..7
    g = vt.Grid.from_u8(vox, pal)
    try:
        g.update((56, 0, 0), np.zeros((8, 8, 16), np.uint8))   # frees slots 6, 7 (bricks 7, 8)
        box = np.zeros((8, 8, 96), np.uint8)                    # bricks 3..14
        box[..., 4 * 8:] = 2                                    # empties 3..6, fills 7..14
        g.update((24, 0, 0), box)
        d, _ = g.bricks()
        assert list(d[1:3]) == [0, 1]
        assert (d[3:7] & 0x80000000).all()
        assert list(d[7:15]) == [5, 4, 3, 2, 7, 6, 8, 9]
        assert g.info()["slots"] == 10
    finally:
        g.destroy()
