"""Edges of the row-strip filter kernel, the one-write integral image and the
per-radius suppression kernel: the tiles' borders, their remainders, unaligned
rows and buffers, and the smallest and largest sizes each takes, bit for bit
against the oracle."""

import ctypes as C

import numpy as np
import pytest

from imageproc_b200 import _lib
from imageproc_b200 import filter as fl
from imageproc_b200 import integral_image as ii
from imageproc_b200 import suppress as sp
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 3, 4])
@pytest.mark.parametrize("kw,kh", [(1, 1), (2, 33), (3, 32), (5, 5), (8, 7), (9, 2)])
def test_filter_strips(channels, kw, kh):
    # 128-element strips of 8 and 32 rows; 8 x 32 taps are the strip kernel's
    # largest, 9 columns or 33 rows the byte tile's
    g = np.random.default_rng(kw * 100 + kh)
    for W, H in ((1, 1), (42, 9), (43, 33), (128, 31), (129, 64), (300, 8)):
        img = g.integers(0, 256, (H, W) if channels == 1 else (H, W, channels), dtype=np.uint8)
        kf = g.standard_normal((kh, kw)).astype(np.float32)
        ki = g.integers(-2**20, 2**20, (kh, kw)).astype(np.int32)
        for k, od in ((kf, np.uint8), (kf, np.float32), (ki, np.int16), (ki, np.int32)):
            got, exp = fl.filter_clamped(img, k, od), O.filter_clamped(img, k, od)
            assert np.array_equal(got.view(np.uint8), exp.view(np.uint8)), (W, H, od)


@pytest.mark.parametrize("channels", [1, 3, 4])
@pytest.mark.parametrize("kw,kh", [(1, 1), (2, 3), (3, 32), (5, 5), (7, 1), (8, 7), (8, 32)])
def test_filter_strips_of_large_images(channels, kw, kh):
    # images that take the strips, in blocks of 8 and of 32 rows: rows on and off
    # word boundaries, one element or row past a block, strips that both ends of
    # a row clamp
    g = np.random.default_rng(kw * 100 + kh)
    for W, H in ((1027, 801), (1152, 797), (129, 8001), (6000, 41), (42, 16003)):
        img = g.integers(0, 256, (H, W) if channels == 1 else (H, W, channels), dtype=np.uint8)
        kf = g.standard_normal((kh, kw)).astype(np.float32)
        ki = g.integers(-2**20, 2**20, (kh, kw)).astype(np.int32)
        for k, od in ((kf, np.uint8), (kf, np.float32), (ki, np.int16), (ki, np.int32)):
            got, exp = fl.filter_clamped(img, k, od), O.filter_clamped(img, k, od)
            assert np.array_equal(got.view(np.uint8), exp.view(np.uint8)), (W, H, od)


def test_filter_large_grid_rows():
    g = np.random.default_rng(3)
    img = g.integers(0, 256, (2051, 2053), dtype=np.uint8)  # 32-row blocks
    k = g.standard_normal((7, 7)).astype(np.float32)
    assert np.array_equal(fl.filter_clamped(img, k, np.uint8), O.filter_clamped(img, k, np.uint8))


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("W,H", [(1, 1), (3, 15), (4, 16), (1023, 17), (1024, 31), (1025, 32), (2049, 33), (5, 700)])
def test_integral_tiles(W, H, dtype):
    g = np.random.default_rng(W + H)
    img = g.integers(0, 256, (H, W), dtype=np.uint8)
    for fn, sq in ((ii.integral_image, False), (ii.integral_squared_image, True)):
        got = fn(img, dtype)
        exp = np.zeros((H + 1, W + 1), np.uint64)
        v = img.astype(np.uint64)
        exp[1:, 1:] = (v * v if sq else v).cumsum(0).cumsum(1)
        assert np.array_equal(got, exp.astype(dtype))


@pytest.mark.parametrize("dtype", [np.uint32, np.uint64])
@pytest.mark.parametrize("W,H", [(4, 1215), (4, 1216), (1024, 1231), (1028, 1283), (2052, 1361), (1, 2000), (3, 2017),
                                 (1023, 2015), (1025, 2401), (2049, 2800)])
def test_integral_strips(W, H, dtype):
    # tall enough for the strips: rows on and off word boundaries, whole and
    # partial last strips, columns at a tile's edges
    test_integral_tiles(W, H, dtype)


def test_integral_unaligned_device_buffers_and_capture():
    # rows off word boundaries, a poisoned table, and the call inside a graph
    import torch
    L = _lib.lib()
    fn = L.ipb_integral_image_device
    fn.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    g = np.random.default_rng(4)
    for off in (0, 1, 2):
        W, H = 1030, 50
        img = g.integers(0, 256, (H, W), dtype=np.uint8)
        buf = torch.zeros(H * W + 8, dtype=torch.uint8, device="cuda")
        d = buf[off:off + H * W]
        d.copy_(torch.from_numpy(img.reshape(-1)))
        out = torch.full((H + 1, W + 1), -1, dtype=torch.int64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _lib.check(fn(d.data_ptr(), W, H, 1, 1, 64, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        graph.replay()
        torch.cuda.synchronize()
        exp = np.zeros((H + 1, W + 1), np.int64)
        exp[1:, 1:] = (img.astype(np.int64) ** 2).cumsum(0).cumsum(1)
        assert np.array_equal(out.cpu().numpy(), exp)


@pytest.mark.parametrize("W,H", [(1, 2001), (2, 2002), (3, 2017), (5, 2017), (1028, 1290), (1030, 2409), (2049, 2801)])
def test_integral_strips_unaligned_device_buffers_and_capture(W, H):
    # tall enough for the strips at every base address: the last words of narrow
    # images, a poisoned table, and the call inside a graph
    import torch
    fn = _lib.lib().ipb_integral_image_device
    fn.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    img = np.random.default_rng(W).integers(0, 256, (H, W), dtype=np.uint8)
    exp = np.zeros((H + 1, W + 1), np.int64)
    exp[1:, 1:] = (img.astype(np.int64) ** 2).cumsum(0).cumsum(1)
    for off in range(4):
        buf = torch.full((H * W + 8,), 255, dtype=torch.uint8, device="cuda")
        d = buf[off:off + H * W]
        d.copy_(torch.from_numpy(img.reshape(-1)))
        out = torch.full((H + 1, W + 1), -1, dtype=torch.int64, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _lib.check(fn(d.data_ptr(), W, H, 1, 1, 64, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), exp), off


@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.uint16, np.int16, np.uint32, np.int32, np.float32])
def test_suppress_every_radius_and_lowest_values(dtype):
    g = np.random.default_rng(np.dtype(dtype).num)
    low = -np.inf if dtype == np.float32 else np.iinfo(dtype).min
    for r in range(0, 18):
        H, W = 33 + r, 129 + 3 * r
        a = g.integers(0, 4, (H, W)).astype(dtype)
        a[: H // 2, : W // 2] = low  # flat regions of the lowest value, the first pixel among them
        got, exp = sp.suppress_non_maximum(a, r), O.suppress_non_maximum(a, r)
        assert np.array_equal(got.view(np.uint8), exp.view(np.uint8)), r
    for a in (np.full((40, 140), low, dtype), np.full((1, 1), low, dtype)):
        assert np.array_equal(sp.suppress_non_maximum(a, 3).view(np.uint8), O.suppress_non_maximum(a, 3).view(np.uint8))
    if dtype == np.float32:
        a = g.standard_normal((50, 150)).astype(np.float32)
        a[3:9, 5:9] = np.frombuffer(b"\xff\xff\xff\xff", np.float32)[0]  # the NaN below every number
        a[20, 40:60] = np.nan
        a[0, 0] = np.frombuffer(b"\xff\xff\xff\xff", np.float32)[0]
        for r in (1, 8, 16):
            assert np.array_equal(sp.suppress_non_maximum(a, r).view(np.uint32),
                                  O.suppress_non_maximum(a, r).view(np.uint32))
