"""The fp32 convolution on the tensor cores: edges of its tiles (128 pixels, 64 and 128 channels, K blocks of 32), every split of
the reduction, every way its activations are loaded, against a double-precision convolution and against the FFMA kernel."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from thnets_b200 import kernels_abi as K  # noqa: E402
from tests import gpu_util as G  # noqa: E402


@pytest.fixture(scope="module")
def lib():
    return K.load()


class Split:
    """A convolution with its weights' parts."""

    def __init__(self, lib, x, wt, stride, pad):
        self.lib, self.x = lib, x
        self.conv = G.Conv(lib, K.THB_F32, x.shape, wt, (stride, stride), (pad, pad))
        d = C.byref(self.conv.d)
        assert lib.thb_conv_f32_supported(d)
        self.parts = G.dzeros(lib.thb_conv_f32_split_bytes(d))
        assert lib.thb_conv_f32_split_weights(d, self.parts.data_ptr(), None) == 0
        self.xt, self.conv.d.in_ld = G.to_nhwc(x, K.THB_F32)

    def run(self, splits, pad=0):
        d = self.conv.d
        d.splits, d.out_ld = splits, G.ru(d.Cout, 4) + pad
        y = torch.full((d.N, d.oH, d.oW, d.out_ld), 3.0, device="cuda")
        rc = self.lib.thb_conv_f32_fwd(C.byref(d), self.parts.data_ptr(), self.xt.data_ptr(), y.data_ptr(), None)
        torch.cuda.synchronize()
        assert rc == 0, (rc, self.lib.thb_last_cuda_error())
        assert int(self.conv.keep[3].cpu()[0]) == 0, "a bounded wait gave up"
        assert pad == 0 or bool((y[..., -pad:] == 3.0).all()), "wrote beyond its channels"
        return G.from_nhwc(y, d.Cout)

    def ffma(self):
        d = self.conv.d
        d.splits, d.out_ld = 0, G.ru(d.Cout, 4)
        return G.from_nhwc(self.conv.run(self.xt), d.Cout)


def double(x, wt, s, p):
    return torch.nn.functional.conv2d(torch.from_numpy(x).double().cuda(), torch.from_numpy(wt).double().cuda(), stride=s, padding=p).cpu().numpy()


CASES = [  # n, cin, h, w, cout, k, stride, pad
    (1, 3, 43, 31, 64, 7, 2, 3),        # gathered, 22 x 16 pixels, K = 196: the last K block a sixth full
    (2, 3, 67, 67, 128, 11, 4, 2),      # gathered, wide tiles
    (1, 16, 9, 9, 64, 3, 1, 1),         # gathered, 16 channels
    (1, 64, 127, 1, 64, 1, 1, 0),       # 127 pixels, a plain matrix of two K blocks: narrow tiles
    (1, 64, 16, 8, 130, 1, 1, 0),       # 128 pixels, channels beyond a tile
    (1, 128, 43, 3, 256, 1, 1, 0),      # 129 pixels, four K blocks: wide tiles
    (3, 64, 9, 5, 200, 3, 2, 1),        # im2col, stride 2, 256 padded channels of 200
    (1, 32, 7, 7, 21, 3, 1, 1),         # im2col, one slab, few channels
    (9, 512, 1, 1, 1000, 1, 1, 0),      # rows of a Linear
    (20, 64, 40, 41, 128, 3, 1, 1),     # more tiles than SMs
    (1, 256, 5, 13, 64, 5, 1, 2),       # 200 K blocks: every ring wraps many times
]


def error(y, ref):
    return np.linalg.norm(y - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("relu", [False, True], ids=["signed", "relu"])
@pytest.mark.parametrize("case", CASES)
def test_tiles_and_splits(lib, case, relu):
    n, cin, h, w, cout, k, s, p = case
    rng = np.random.default_rng(cin + k)
    x = rng.standard_normal((n, cin, h, w)).astype(np.float32)
    if relu:
        x = np.maximum(x, 0)
    wt = (rng.standard_normal((cout, cin, k, k)) * (cin * k * k) ** -0.5).astype(np.float32)
    ref = double(x, wt, s, p)
    c = Split(lib, x, wt, s, p)
    before = error(c.ffma(), ref)
    for splits in (0, 1, 2, 4, 8):
        y = c.run(splits, pad=4)
        # never further from the exact result than the FFMA kernel: measured 6.0e-8 to 2.3e-7 against 7.8e-8 to 4.3e-7
        assert error(y, ref) <= before, splits
        assert G.rel_err(y, ref) < 1e-6, splits
        assert np.array_equal(y, c.run(splits)), splits
    # residual, scale, shift and the activations
    scale, shift = rng.uniform(0.5, 1.5, cout).astype(np.float32), rng.standard_normal(cout).astype(np.float32)
    res = rng.standard_normal(ref.shape).astype(np.float32)
    c.conv.set_affine(scale, shift)
    rt, rld = G.to_nhwc(res, K.THB_F32)
    c.conv.set_residual(rt, rld, 1.0, -1.0)
    want = ref * scale[None, :, None, None] + shift[None, :, None, None] - res
    slope = rng.uniform(0.1, 0.5, cout).astype(np.float32)
    for kind, kw, f in ((K.ACT_THRESHOLD, dict(threshold=0.1, value=-1.0), lambda v: np.where(v > 0.1, v, -1.0)),
                        (K.ACT_PRELU, dict(slope=slope), lambda v: np.where(v > 0, v, v * slope[None, :, None, None]))):
        c.conv.set_act(kind, **kw)
        for splits in (1, 4):
            y, keep = c.run(splits), np.abs(want - 0.1) > 1e-5  # (a value at the threshold may fall on either side)
            assert G.rel_err(np.where(keep, y, 0), np.where(keep, f(want), 0)) < 1e-6, (kind, splits)


def test_values_the_parts_cannot_hold(lib):
    """Infinities, NaN and values near the end of fp32's range come out as the FFMA kernel has them."""
    rng = np.random.default_rng(5)
    x = rng.standard_normal((1, 64, 12, 12)).astype(np.float32)
    wt = (rng.standard_normal((64, 64, 3, 3)) * 0.1).astype(np.float32)
    wt[:, 1] = 0.5      # parts beyond the first are zero: infinity times them would be NaN
    wt[:, 2] = 0.0      # 0 x infinity is NaN in the reference's order of operations as well
    x[0, 1, 2, 2], x[0, 1, 8, 8], x[0, 3, 2, 9], x[0, 2, 9, 2] = np.inf, -np.inf, np.nan, np.inf
    x[0, 4, 5, 5] = 3.4e38  # rounds to an infinite bf16
    wt[:, 4] = 0.25
    c = Split(lib, x, wt, 1, 1)
    a = c.ffma()
    assert np.isinf(a).any() and np.isnan(a).any() and np.isfinite(a).any() and (np.abs(a[np.isfinite(a)]) > 1e37).any()
    for splits in (1, 2, 8):
        b = c.run(splits)
        assert np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(np.isinf(a), np.isinf(b)), splits
        same = np.isinf(a)
        assert np.array_equal(a[same], b[same])
        fin = np.isfinite(a)
        assert np.abs(a[fin] / b[fin] - 1).max() < 1e-3 and G.rel_err(b[fin], a[fin]) < 1e-6


SHAPES = [(1, 64, 12, 12, 64, 3, 1, 1), (1, 128, 9, 9, 128, 1, 1, 0), (1, 3, 20, 20, 128, 7, 2, 3)]  # im2col, matrix (wide tiles), gathered
SCALES = [(1e-20, 1), (1e-30, 1), (1e-33, 1), (1e-35, 1), (1e-37, 1), (1e-40, 1), (1e-43, 1), (1, 1e-30), (1, 1e-35), (1, 1e-37), (1, 1e-41),
          (1e-20, 1e-15), (1e-20, 1e-19), (1e10, 1e-40), (1e25, 1e-37), (1e-37, 1e20), (1e30, 1e-33), (1e-38, 1e37), (1e30, 1e-43)]


def no_worse(c, ref, shape):
    """Every split's result is as near to the exact one as the FFMA kernel's, but for the last bits of fp32's smallest numbers: a product
    and its addition round by half of 2^-149, once for each of the K products and once more for each of their sums of 32."""
    _, cin, _, _, _, k, _, _ = shape
    before, quantum = error(c.ffma(), ref), 2.0 ** -150 * cin * k * k * 33 / 32
    for splits in (0, 1, 2, 8):
        y = c.run(splits)
        small = np.abs(ref) < 2.0 ** -110
        assert not small.any() or (np.abs(y - ref) <= 1e-6 * np.abs(ref).max() + quantum)[small].all(), splits
        assert np.abs(ref).max() < 2.0 ** -110 or error(y, ref) <= before, splits


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("xs,ws", SCALES)
def test_magnitudes(lib, shape, xs, ws):
    """Values of any size keep their bits, down to where bf16 has none left."""
    n, cin, h, w, cout, k, s, p = shape
    rng = np.random.default_rng(cin)
    x = (rng.standard_normal((n, cin, h, w)) * xs).astype(np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) * 0.1 * ws).astype(np.float32)
    c = Split(lib, x, wt, s, p)
    no_worse(c, double(x, wt, s, p), shape)


@pytest.mark.parametrize("shape", SHAPES)
def test_mixed_magnitudes(lib, shape):
    """Tiny values beside large ones: in a row of activations, in a channel of weights, between the channels; sums that are zero."""
    n, cin, h, w, cout, k, s, p = shape
    rng = np.random.default_rng(cin + 1)
    x0 = rng.standard_normal((n, cin, h, w)).astype(np.float32)
    w0 = (rng.standard_normal((cout, cin, k, k)) * 0.1).astype(np.float32)
    zeros = np.zeros_like(x0)
    zeros[:, cin // 2, h // 2, w // 2] = 1e-42    # alone: a row whose every product vanishes
    zeros[:, cin // 2, 0, 0] = 1e-36
    c = Split(lib, zeros, w0, s, p)
    no_worse(c, double(zeros, w0, s, p), shape)
    wide = w0 * np.float32(1e-37)
    wide[:, 0] = 1                                # the channels' largest weights meet zeros
    wide[1::2] *= np.float32(1e-3)
    for xs in (1, 1e20, 1e37):
        x = x0 * np.float32(xs)
        x[:, 0] = 0
        c = Split(lib, x, wide, s, p)
        no_worse(c, double(x, wide, s, p), shape)
    apart = w0 * (10.0 ** rng.uniform(-44, 10, (cout, 1, 1, 1)))  # channels of all sizes, one of them zero
    apart[3] = 0
    apart = apart.astype(np.float32)
    c = Split(lib, x0, apart, s, p)
    ref, rounding = double(x0, apart, s, p), 2.0 ** -150 * cin * k * k * 33 / 32
    scale = (10.0 ** rng.uniform(-40, 3, cout)).astype(np.float32)
    for sc in (np.ones(cout, np.float32), scale):
        c.conv.set_affine(sc, None)
        want, before = ref * sc[None, :, None, None], c.ffma()
        for splits in (1, 2, 8):
            y = c.run(splits)
            for o in range(cout):
                bound = 1e-6 * np.abs(want[:, o]).max() + rounding * sc[o] + 2.0 ** -150
                assert np.abs(y[:, o] - want[:, o]).max() <= max(np.abs(before[:, o] - want[:, o]).max(), bound), (splits, o)


def test_bounded_wait(lib, monkeypatch):
    """A copy that is never made: the launch ends, reports, and the next one is right."""
    rng = np.random.default_rng(6)
    x = rng.standard_normal((1, 64, 10, 10)).astype(np.float32)
    wt = rng.standard_normal((64, 64, 3, 3)).astype(np.float32)
    c = Split(lib, x, wt, 1, 1)
    good = c.run(2)
    monkeypatch.setenv("THB200_TEST_WITHHOLD", "1")
    monkeypatch.setenv("THB200_WAIT_LIMIT_CYCLES", "20000000")
    lib.thb_conv_reload_knobs()
    try:
        y = torch.zeros((1, 10, 10, 64), device="cuda")
        for splits in (1, 2):
            c.conv.d.splits = splits
            assert lib.thb_conv_f32_fwd(C.byref(c.conv.d), c.parts.data_ptr(), c.xt.data_ptr(), y.data_ptr(), None) == 0
            torch.cuda.synchronize()
            assert int(c.conv.keep[3].cpu()[0]) != 0
            c.conv.keep[3].zero_()
    finally:
        monkeypatch.undo()
        lib.thb_conv_reload_knobs()
    assert np.array_equal(c.run(2), good)


@pytest.mark.parametrize("n,cin,side,cout,k", [(16, 1024, 14, 256, 1), (16, 128, 28, 128, 3), (4, 256, 56, 64, 1)])
def test_cold_activations(lib, n, cin, side, cout, k):
    """Activations from memory, of which some K blocks arrive late and out of order: every launch gives the same bits, and no wait runs
    out.  (A wide net: a ring whose stages change between the splitting groups, which the kernel's assertions rule out, failed once in
    thousands of launches.)"""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((n, cin, side, side)).astype(np.float32)
    c = Split(lib, x, (rng.standard_normal((cout, cin, k, k)) / (cin * k * k) ** 0.5).astype(np.float32), 1, k // 2)
    big = torch.empty(160 << 20, dtype=torch.uint8, device="cuda")
    c.run(0)
    d = c.conv.d
    first, y = (torch.zeros((n, side, side, d.out_ld), device="cuda") for _ in range(2))
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(1500):
        big.fill_(i & 255)
        out = y if i else first
        assert lib.thb_conv_f32_fwd(C.byref(d), c.parts.data_ptr(), c.xt.data_ptr(), out.data_ptr(), None) == 0
        if i:
            differ += (y != first).any()
    assert int(c.conv.keep[3].cpu()[0]) == 0, "a bounded wait gave up"
    assert int(differ) == 0 and bool(torch.isfinite(first).all())


@pytest.mark.parametrize("cin,h,w,cout,k,s,p", [(3, 67, 67, 128, 11, 4, 2), (128, 43, 3, 256, 1, 1, 0), (64, 9, 9, 128, 3, 1, 1), (64, 9, 9, 200, 5, 1, 2)])
def test_half_tiles(lib, cin, h, w, cout, k, s, p):
    """Layers of 128 channels a tile: few tiles go to CTAs of 64 channels, which read halves of the weights' stages.  The K blocks and
    their order are the same, so an image gives the same bits in a launch of either kind."""
    rng = np.random.default_rng(cout + k)
    x = rng.standard_normal((1, cin, h, w)).astype(np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) * (cin * k * k) ** -0.5).astype(np.float32)
    one = Split(lib, x, wt, s, p)
    d = one.conv.d
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = -(-d.oH * d.oW // 128) * (d.Cout_pad // 64)
    assert d.Cout_pad % 128 == 0 and tiles * 16 <= sms
    n = -(-(sms + 1) * 64 * 128 // (d.Cout_pad * d.oH * d.oW)) + 1
    many = Split(lib, np.repeat(x, n, 0), wt, s, p)
    ref = double(x, wt, s, p)
    bound = error(one.ffma(), ref)
    for splits in (1, 2, 4, 8):
        y = one.run(splits, pad=4)
        assert error(y, ref) <= bound, splits
        wide = many.run(splits)
        assert np.array_equal(wide[:1], y) and np.array_equal(wide[-1:], y), splits
