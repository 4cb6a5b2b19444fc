"""The convolution kernel for launches of few tiles (conv_few_tc.cu): every split, ragged rows and channels, every operand
mode, against an fp32 convolution of the same rounded inputs -- and, unsplit, against the persistent kernel bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from thnets_b200 import kernels_abi as K  # noqa: E402
from tests import gpu_util as G  # noqa: E402


@pytest.fixture(scope="module")
def lib():
    lib = K.load()
    lib.thb_conv_few_supported.argtypes = [C.c_void_p]
    return lib


def rounded(a, dtype):
    t = torch.float16 if dtype == K.THB_F16 else torch.bfloat16
    return torch.from_numpy(a).to(t).float()


CASES = [  # n, cin, h, w, cout, k, stride, pad
    (1, 512, 7, 7, 512, 3, 1, 1),     # one row tile, mostly ragged
    (1, 64, 9, 15, 64, 1, 1, 0),      # 135 rows: a second tile of 7; one K block
    (2, 128, 8, 8, 72, 1, 1, 0),      # exactly one row tile, ragged channels
    (3, 64, 11, 13, 200, 3, 2, 1),    # stride, 4 channel tiles, the last ragged
    (1, 256, 5, 6, 66, 5, 1, 2),
    (9, 192, 1, 1, 1000, 1, 1, 0),    # a Linear
    (2, 64, 57, 31, 64, 3, 1, 1),
    (20, 64, 45, 43, 72, 1, 1, 0),    # 606 tiles: the form with four epilogue warps
]


@pytest.mark.parametrize("dtype", [K.THB_F16, K.THB_BF16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("case", CASES)
def test_few_tiles(lib, case, dtype, monkeypatch):
    n, cin, h, w, cout, k, s, p = case
    rng = np.random.default_rng(7)
    x = rounded(rng.standard_normal((n, cin, h, w)).astype(np.float32), dtype)
    wt = rounded((rng.standard_normal((cout, cin, k, k)) * (cin * k * k) ** -0.5).astype(np.float32), dtype)
    scale, shift = rng.uniform(0.5, 1.5, cout).astype(np.float32), rng.standard_normal(cout).astype(np.float32)
    slope = rng.uniform(0.1, 0.3, cout).astype(np.float32)
    ref = torch.nn.functional.conv2d(x.double().cuda(), wt.double().cuda(), stride=s, padding=p).cpu().numpy()
    ref = ref * scale[None, :, None, None] + shift[None, :, None, None]
    res = rounded(rng.standard_normal(ref.shape).astype(np.float32), dtype).numpy()
    want = {"plain": ref, "relu+res": np.maximum(ref - res, 0), "prelu": np.where(ref > 0, ref, ref * slope[None, :, None, None])}
    xt, _ = G.to_nhwc(x.numpy(), dtype)
    nkb = k * k * cin // 64

    def run(kind, splits, few=True):
        monkeypatch.setenv("THB200_FEW_TILES", "100000" if few else "0")
        monkeypatch.setenv("THB200_NO_PATCH", "1")
        lib.thb_conv_reload_knobs()
        conv = G.Conv(lib, dtype, x.shape, wt.numpy(), (s, s), (p, p), bn_tile=64)
        conv.set_affine(scale, shift, host_copies=True)
        if kind == "relu+res":
            rt, rld = G.to_nhwc(res, dtype)
            conv.set_residual(rt, rld, 1.0, -1.0)
            conv.set_act(K.ACT_THRESHOLD)
        elif kind == "prelu":
            conv.set_act(K.ACT_PRELU, slope=slope)
        conv.d.splits = splits
        assert lib.thb_conv_few_supported(C.byref(conv.d)) == int(few)
        y = conv.run(xt, out_ld=G.ru(cout, 8) + 8, fill=3.0)
        assert bool((y[..., G.ru(cout, 8):] == 3.0).all()), "wrote beyond its channels"
        if cout % 8:
            assert bool((y[..., cout:G.ru(cout, 8)] == 0).all()), "padded channels must be zero"
        return G.from_nhwc(y, cout)

    tol = 2e-3 if dtype == K.THB_F16 else 1e-2
    try:
        for kind in want:
            for splits in (1, 2, 4, 8):
                if splits > 1 and nkb < splits:
                    continue
                out = run(kind, splits)
                assert G.rel_err(out, want[kind]) < tol, (kind, splits)
                if splits == 1:
                    assert np.array_equal(out, run(kind, 0, few=False)), kind
                else:
                    assert np.array_equal(out, run(kind, splits)), (kind, splits)
    finally:
        monkeypatch.undo()
        lib.thb_conv_reload_knobs()


@pytest.mark.parametrize("splits", [1, 4])
def test_bounded_wait(lib, splits, monkeypatch):
    """A copy that is never made: the launch ends (the peers of the CTA that lacks it give up their own waits), reports, and the next
    one is right."""
    rng = np.random.default_rng(6)
    conv = G.Conv(lib, K.THB_F16, (1, 64, 10, 10), rng.standard_normal((64, 64, 3, 3)).astype(np.float32), (1, 1), (1, 1))
    conv.d.splits = splits
    xt, _ = G.to_nhwc(rng.standard_normal((1, 64, 10, 10)).astype(np.float32), K.THB_F16)
    monkeypatch.setenv("THB200_FEW_TILES", "100000")
    monkeypatch.setenv("THB200_NO_PATCH", "1")
    try:
        lib.thb_conv_reload_knobs()
        good = conv.run(xt)
        monkeypatch.setenv("THB200_TEST_WITHHOLD", "1")
        monkeypatch.setenv("THB200_WAIT_LIMIT_CYCLES", "20000000")
        lib.thb_conv_reload_knobs()
        y = torch.zeros_like(good)
        assert lib.thb_conv_fwd(C.byref(conv.d), G.ptr(xt), G.ptr(y), None) == 0
        torch.cuda.synchronize()
        assert int(conv.keep[3].cpu()[0]) != 0
        conv.keep[3].zero_()
    finally:
        monkeypatch.undo()
        lib.thb_conv_reload_knobs()
    monkeypatch.setenv("THB200_FEW_TILES", "100000")
    lib.thb_conv_reload_knobs()
    try:
        assert torch.equal(conv.run(xt), good)
    finally:
        monkeypatch.undo()
        lib.thb_conv_reload_knobs()


@pytest.mark.parametrize("dtype", [K.THB_F16, K.THB_BF16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("case", [(2, 48, 12, 20, 21, 1, 1, 0), (1, 64, 9, 15, 70, 3, 1, 1), (3, 128, 8, 16, 33, 1, 1, 0)])
def test_result_as_nchw_floats(lib, case, dtype):
    """A last convolution that leaves NCHW floats: the bits of the 16-bit result, transposed and widened."""
    n, cin, h, w, cout, k, s, p = case
    rng = np.random.default_rng(3)
    x = rounded(rng.standard_normal((n, cin, h, w)).astype(np.float32), dtype).numpy()
    wt = rounded((rng.standard_normal((cout, cin, k, k)) * (cin * k * k) ** -0.5).astype(np.float32), dtype).numpy()
    conv = G.Conv(lib, dtype, x.shape, wt, (s, s), (p, p))
    conv.set_affine(rng.uniform(0.5, 1.5, cout), rng.standard_normal(cout), host_copies=True)
    conv.set_act(K.ACT_THRESHOLD)
    xt, _ = G.to_nhwc(x, dtype)
    want = G.from_nhwc(conv.run(xt), cout)
    out, status = torch.zeros(want.shape, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    lib.thb_conv_nchw_fwd.argtypes = [C.c_void_p] * 5
    assert lib.thb_conv_nchw_fwd(C.byref(conv.d), G.ptr(xt), G.ptr(out), G.ptr(status), None) == 0
    torch.cuda.synchronize()
    assert int(status[0]) == 0 and np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("net,size,batch", [("resnet18", 64, 1), ("resnet18", 97, 3), ("resnet50", 64, 2), ("resnet50", 161, 1), ("vgg16", 64, 2)])
@pytest.mark.parametrize("images", [True, False], ids=["bytes", "floats"])
def test_uint8_networks(lib, tmp_path, monkeypatch, net, size, batch, images):
    """uint8 networks whose layers are a few tiles each (3x3, 1x1, strided, half-block taps, residuals, Linear layers; clusters
    of 1 to 8): the bytes of the persistent kernel."""
    from thnets_b200 import fixtures as fx
    from thnets_b200.capi import THNets
    th = THNets()
    g = fx.vgg16(size=size, classes=37, fc=200) if net == "vgg16" else getattr(fx, net)(size=size, classes=37, fc_bias=0.05)
    path = str(tmp_path / "n.net")
    fx.write_pymodel(g, path)
    rng = np.random.default_rng(size)
    x = [rng.integers(0, 256, (size, size, 3), dtype=np.uint8) for _ in range(batch)] if images else g.make_input(batch)
    outs = []
    try:
        for few in (None, "0"):
            if few:
                monkeypatch.setenv("THB200_FEW_TILES", few)
            lib.thb_conv_reload_knobs()
            h = th.load_network(path)
            th.set_stats(h, (0.45,) * 3, (0.225,) * 3)
            handle = th.create_lowp_network(h, 20.0)
            th.free_network(h)
            outs += [(th.process_images(handle, x) if images else th.process_float(handle, x))[0] for _ in range(3)]
            th.free_network(handle)
    finally:
        monkeypatch.undo()
        lib.thb_conv_reload_knobs()
    assert outs[0].std() > 0
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
