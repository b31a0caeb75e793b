"""Directory distances of small lattices with bricks that have no occupied brick within 14: nothing
occupied at all, at 15 bricks along an axis (every brick in reach of every other: the cap without the
distance passes) and at 16 and more, in the one-block, the graph and the general build, and updates that
empty such a grid and fill one corner again.  Whole numbers: equal to the brute-force restatement."""
import numpy as np
import pytest

import vtrace_gb300 as vt
from test_gpu_parity import expected_bricks, expected_long, expected_octants

pytestmark = pytest.mark.gpu


def check(g, vox, pal, dims):
    d, _ = g.bricks()
    want = expected_bricks(vox, pal)[0]
    empty = want >> 31 == 1
    np.testing.assert_array_equal(d >> 31, want >> 31)
    np.testing.assert_array_equal(d[empty], want[empty])
    oc = g.octants()
    np.testing.assert_array_equal(oc, expected_octants(d, dims))
    np.testing.assert_array_equal(g.long_boxes(), expected_long(d, oc, dims))


# bricks: 15, 16 and 32 in a row (one block), 5 x 6 x 15, 5 x 6 x 16 (graph), 15^3, 16 x 15 x 15 (general)
@pytest.mark.parametrize("dims", [(15 * 8, 8, 8), (8, 16 * 8 - 7, 8), (8, 8, 32 * 8), (40, 48, 120), (121, 40, 41),
                                  (120, 113, 120), (113, 121, 120)])
@pytest.mark.parametrize("corner", [False, True])
def test_distances_of_small_lattices(dims, corner):
    pal = vt.gen_palette(3)
    vox = np.zeros(dims[::-1], np.uint8)
    if corner:
        vox[0, 0, -1] = 4
    g = vt.Grid.from_u8(vox, pal)
    try:
        check(g, vox, pal, dims)
        for value in (0, 5):  # the corner emptied, then the opposite one filled
            at = (0, 0, dims[0] - 1) if value == 0 else (dims[2] - 1, dims[1] - 1, 0)
            vox[at] = value
            g.update(at[::-1], np.full((1, 1, 1), value, np.uint8))
            check(g, vox, pal, dims)
    finally:
        g.destroy()
