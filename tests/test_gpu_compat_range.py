"""render_tick instances whose matrices lie near the ends of binary32's range, where the approximate
arithmetic of the culling and of the slab test leaves it: a plate 3e-39 thick, whose inverse has elements of
3e38 (the reciprocals of a ray's components in it are subnormal), and a floor 3e37 long seen through a
narrow projection (its far corners' products overflow).  Every pixel equals the oracle's loop over every
instance."""
import ctypes
import math
import struct

import numpy as np
import pytest

import vtrace_gb300 as vt
from oracle import pyoracle as po
from test_gpu_compat import instance, lib, look_at, perspective  # noqa: F401 (lib: a fixture)

pytestmark = pytest.mark.gpu

W, H = 96, 64


def check(lib, monkeypatch, textures, insts, P, C):  # noqa: F811
    monkeypatch.setenv("VTRACE_WIDTH", str(W))
    monkeypatch.setenv("VTRACE_HEIGHT", str(H))
    insts = np.ascontiguousarray(np.stack(insts))
    assert lib.entry() == 0
    try:
        for t in textures:
            assert lib.add_texture(t.ctypes.data, 8, 8, 8) >= 0
        ptr = lib.start_update_instances(len(insts))
        ctypes.memmove(ptr, insts.ctypes.data, insts.nbytes)
        assert lib.end_update_instances(len(insts)) == 0
        info = vt.RenderTickInfo(P.ctypes.data, C.ctypes.data)
        ww, hh = ctypes.c_int32(0), ctypes.c_int32(0)
        assert lib.render_tick(ctypes.byref(ww), ctypes.byref(hh), ctypes.byref(info)) == 0
        fb = np.zeros((H, W, 4), np.uint8)
        assert lib.vt_framebuffer_download(fb.ctypes.data, fb.nbytes) == 0
    finally:
        lib.cleanup()
    want = po.compat_render([po.Grid(texels=t) for t in textures], insts, P.reshape(16), C.reshape(16), W, H)
    diff = np.nonzero((fb != want).any(-1))
    assert len(diff[0]) == 0, (len(diff[0]), diff[0][:5], diff[1][:5])
    assert (want != np.array([0xC0, 0xE8, 0xF6, 0xFF], np.uint8)).any(-1).sum() >= 99


PLATE = np.full((8, 8, 8), 0xFF2040C0, np.uint32)
BLOCK = np.full((8, 8, 8), 0xFF30C040, np.uint32)


@pytest.mark.parametrize("scale", [(3e-39, 0.8, 0.8), (0.8, 3e-39, 0.8), (0.8, 0.8, 3e-39), (1e-38, 0.8, 0.8),
                                   (3e-39, 3e-39, 2)])
def test_thin_instances_equal_the_oracle(lib, monkeypatch, scale):  # noqa: F811
    insts = [instance(0, (0, 1, 0), scale, (0, 0, -0.3), 0),
             instance(25, (1, 1, 0), (0.5, 0.5, 0.5), (0.2, -0.3, -1.2), 1),
             instance(0, (0, 1, 0), scale, (-0.2, 0.1, -0.35), 0)]
    check(lib, monkeypatch, [PLATE, BLOCK], insts, perspective(math.radians(80.0), W / H, 0.01, 200.0),
          look_at((0.4, 0.3, 0.5), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0)))


@pytest.mark.parametrize("side", [-2e33, 2e33])
@pytest.mark.parametrize("far", [1.5e37, 2e37])
def test_huge_instances_equal_the_oracle(lib, monkeypatch, side, far):  # noqa: F811
    fov, near = math.radians(2.0), 3e35
    f, r, up = np.array([1, 0, -1]) / math.sqrt(2), np.array([1, 0, 1]) / math.sqrt(2), np.array([0, 1, 0])
    k = math.tan(fov / 2) * W / H
    a, b = (f * z + r * (z * k * xn) + up * side for z, xn in ((near, -0.8), (far, 0.8)))
    M = np.eye(4)
    M[:3] = np.stack([b - a, up * 1e22, r * (k * 0.3 * near), (a + b) / 2], 1)
    cm = np.ascontiguousarray(M.T, np.float32).reshape(16)
    cm[15] = struct.unpack("<f", struct.pack("<i", 0))[0]
    check(lib, monkeypatch, [PLATE], [cm], perspective(fov, W / H, 0.01, 200.0),
          look_at((0, 0, 0), (1, 0, -1), (0, 1, 0)))
