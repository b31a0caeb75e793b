"""Slots, masks, payloads and directory of builds against a restatement with numpy: lattices of a group of
32 bricks less one, one and one more, groups with 0 to 32 occupied bricks, the brick counts where the
compaction stops splitting a group over warps (2,047 and 2,048 groups), partial bricks, both formats, and the
build into the caller's buffers."""
import numpy as np
import pytest

import vtrace_gb300 as vt

pytestmark = pytest.mark.gpu


def lattice(dims, seed):
    """Voxels whose bricks are occupied in runs: groups of 32 from empty to full."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    b = tuple((n + 7) // 8 for n in (nz, ny, nx))
    n = b[0] * b[1] * b[2]
    share = np.repeat(rng.choice([0.0, 0.03, 0.5, 1.0], (n + 31) // 32), 32)[:n]
    full = (rng.random(n) < share).reshape(b)
    # one to three occupied voxels in an occupied brick: the first always, so that partial bricks have it
    bricks = np.zeros((n, 512), np.uint8)
    bricks[:, 0] = rng.integers(1, 256, n)
    for _ in range(2):
        bricks[np.arange(n), rng.integers(0, 512, n)] = rng.integers(1, 256, n)
    bricks[~full.reshape(-1)] = 0
    vox = bricks.reshape(b + (8, 8, 8)).transpose(0, 3, 1, 4, 2, 5).reshape(b[0] * 8, b[1] * 8, b[2] * 8)
    return np.ascontiguousarray(vox[:nz, :ny, :nx])


def expected(vox):
    nz, ny, nx = vox.shape
    b = tuple((n + 7) // 8 for n in vox.shape)
    pad = np.zeros(tuple(8 * k for k in b), np.uint8)
    pad[:nz, :ny, :nx] = vox
    bricks = pad.reshape(b[0], 8, b[1], 8, b[2], 8).transpose(0, 2, 4, 1, 3, 5).reshape(-1, 512)
    full = bricks.any(1)
    payload = bricks[full]
    masks = np.packbits(payload.reshape(-1, 8, 64) != 0, axis=2, bitorder="little").view(np.uint64)[..., 0]
    slots = np.cumsum(full, dtype=np.int64) - 1
    return full, slots, masks, payload


def same(directory, masks, payload, want):
    full, slots, w_masks, w_payload = want
    np.testing.assert_array_equal(directory >> 31 == 0, full)
    np.testing.assert_array_equal(directory[full], slots[full])
    np.testing.assert_array_equal(masks[:len(w_masks)], w_masks)
    np.testing.assert_array_equal(payload[:len(w_payload)].reshape(-1, 512), w_payload)


@pytest.mark.parametrize("dims", [(65 * 8, 8, 8), (95 * 8, 8, 8), (8, 96 * 8, 8), (8, 8, 97 * 8), (83, 75, 61), (250, 255, 131),
                                  (89 * 8, 736 * 8, 8), (2048, 2041, 3)])
def test_builds_match_the_restatement(dims):
    vox = lattice(dims, sum(dims))
    want = expected(vox)
    pal = vt.gen_palette(3)
    g = vt.Grid.from_u8(vox, pal)
    try:
        d, m = g.bricks()
        same(d, m, g.payload(), want)
        assert g.info()["voxels_occupied"] == np.count_nonzero(vox)
    finally:
        g.destroy()
    if vox.size <= 1 << 24:
        g = vt.Grid.from_rgba8(np.where(vox != 0, 0xFF000000 | vox.astype(np.uint32), 0).astype(np.uint32))
        try:
            d, m = g.bricks()
            same(d, m, np.ascontiguousarray(g.payload()[..., 0]), want)
        finally:
            g.destroy()


@pytest.mark.parametrize("dims", [(8, 8, 8), (31 * 8, 8, 8), (8, 32 * 8, 8), (8, 8, 33 * 8), (83, 75, 61), (256, 255, 256)])
def test_builds_into_the_callers_buffers_match_the_restatement(dims):
    import torch
    assert torch.cuda.is_available()
    vt.init(0)
    vox = lattice(dims, sum(dims))
    want = expected(vox)
    n = len(want[0])
    pal = torch.from_numpy(vt.gen_palette(3).view(np.uint8)).cuda()
    src = torch.from_numpy(vox.reshape(-1)).cuda()
    d, m, p, c = (torch.full((k,), 0xAB, dtype=torch.uint8, device="cuda") for k in (n * 4, n * 64, n * 512, 16))
    assert vt.lib().vt_grid_build_u8_noalloc(src.data_ptr(), pal.data_ptr(), *dims, d.data_ptr(), m.data_ptr(),
                                             p.data_ptr(), c.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    same(d.cpu().numpy().view(np.uint32), m.cpu().numpy().view(np.uint64).reshape(-1, 8), p.cpu().numpy().reshape(-1, 512), want)
    assert list(c.cpu().numpy().view(np.uint64)) == [int(want[0].sum()), int(np.count_nonzero(vox))]
