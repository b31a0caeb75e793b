"""Empty-space tables (directory distances, octant and long-box words) at the sizes where the lattice
passes change course: 32-brick words and 8-row tiles with remainders on every axis, lattices one
brick thick, bricks farther than 14 from every occupied one (distances 15..31 come from passes of
their own), and updates that make such bricks appear, move and vanish.  The tables are whole numbers:
equality with the brute-force restatements, and of an updated grid with a fresh build."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from test_gpu_parity import expected_bricks, expected_long, expected_octants
from test_gpu_update import same_as_fresh

pytestmark = pytest.mark.gpu


def points(rng, dims, count):
    vox = np.zeros(dims[::-1], np.uint8)
    for _ in range(count):
        vox[tuple(int(rng.integers(0, n)) for n in vox.shape)] = int(rng.integers(1, 256))
    return vox


@pytest.mark.parametrize("dims,count", [
    ((33 * 8, 9 * 8 - 3, 17 * 8), 40),     # one brick past a word, one row past a tile
    ((9 * 8, 33 * 8, 31 * 8 + 1), 60),
    ((65 * 8, 8, 24), 3),                  # thin lattices, distances up to the cap
    ((8, 70 * 8, 16), 2),
    ((20, 9, 66 * 8), 2),
    ((40 * 8, 36 * 8, 33 * 8), 2),         # distances 15..31 along every axis
    ((34 * 8, 34 * 8, 34 * 8), 0),         # nothing occupied
])
def test_tables_match_brute_force(dims, count):
    vox = points(np.random.default_rng(sum(dims) + count), dims, count)
    pal = vt.gen_palette(3)
    g = vt.Grid.from_u8(vox, pal)
    try:
        d, _ = g.bricks()
        np.testing.assert_array_equal(d, expected_bricks(vox, pal)[0])
        oc = g.octants()
        np.testing.assert_array_equal(oc, expected_octants(d, dims))
        np.testing.assert_array_equal(g.long_boxes(), expected_long(d, oc, dims))
    finally:
        g.destroy()


@pytest.mark.parametrize("dims,count", [((280, 264, 300), 3), ((520, 24, 40), 4), ((300, 290, 64), 200)])
def test_updates_match_fresh_builds(dims, count):
    rng = np.random.default_rng(sum(dims))
    vox, pal = points(rng, dims, count), vt.gen_palette(5)
    g = vt.Grid.from_u8(vox, pal)
    try:
        for step in range(6):
            size = [min(n, s) for n, s in zip(dims, (16, 16, 16) if step % 2 else (150, 170, 131))]
            x, y, z = (int(rng.integers(0, n - s + 1)) for n, s in zip(dims, size))
            box = np.zeros(size[::-1], np.uint8)  # a large box cleared, then a small one filled
            if step % 2:
                box[rng.random(box.shape) < 0.02] = 7
            vox[z:z + size[2], y:y + size[1], x:x + size[0]] = box
            g.update((x, y, z), box)
            fresh = vt.Grid.from_u8(vox, pal)
            try:
                same_as_fresh(g, fresh)
            finally:
                fresh.destroy()
    finally:
        g.destroy()
