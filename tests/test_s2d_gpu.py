"""First convolutions of stride 2 and 4 on a space-to-depth input (any side lengths, floats and byte pictures, one picture or
a batch) against the same network with the layer as it is: uint8 bit for bit, 16-bit types up to the order of the sums."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests import gpu_util as G
from thnets_b200 import fixtures as fx
from thnets_b200 import kernels_abi as K
from thnets_b200.capi import THNets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def th():
    return THNets()


def forward(th, path, mode, x, images, monkeypatch, s2d):
    monkeypatch.setenv("THB200_NO_S2D", "0" if s2d else "1")
    h = th.load_network(path)
    th.set_stats(h, (0.45, 0.4, 0.5), (0.225, 0.25, 0.2))
    if mode == 3:
        net = th.create_lowp_network(h, 8.0)
    else:
        th.lib.THB200_SetPrecision(mode)
        net = th.lib.THCreateCudaNetwork(h)
        th.lib.THB200_SetPrecision(0)
    assert net
    th.free_network(h)
    if images:
        out = th.process_images(net, x)[0]
    else:
        before = x.copy()
        out = th.process_float(net, x, copy_input=False)[0]
        norm = (before - np.float32([0.45, 0.4, 0.5])[:, None, None]) / np.float32([0.225, 0.25, 0.2])[:, None, None]
        assert np.array_equal(x, norm.astype(np.float32)), "the in-place side effect"
        x[...] = before
    th.free_network(net)
    return out


@pytest.mark.parametrize("mode", [1, 2, 3], ids=["fp16", "bf16", "uint8"])
@pytest.mark.parametrize("images", [True, False], ids=["bytes", "floats"])
@pytest.mark.parametrize("k,stride,pad", [(7, 2, 3), (3, 2, 1), (5, 2, 0), (11, 4, 2), (4, 4, 0)])
@pytest.mark.parametrize("n,h,w", [(1, 33, 40), (3, 32, 47), (2, 31, 29), (1, 64, 64)])
def test_first_layer(th, tmp_path, monkeypatch, mode, images, k, stride, pad, n, h, w):
    g = fx.Graph(3)
    g.input_shape = (3, h, w)
    x = g.relu(g.conv(0, 3, 40, k, stride, pad, bias=0.1))
    g.conv(x, 40, 24, 1, 1, 0, bias=0.1)
    path = str(tmp_path / "n.net")
    fx.write_pymodel(g, path)
    rng = np.random.default_rng(k * h + w)
    x = [rng.integers(0, 256, (h, w, 3), dtype=np.uint8) for _ in range(n)] if images else rng.random((n, 3, h, w), dtype=np.float32)
    a = forward(th, path, mode, x, images, monkeypatch, True)
    b = forward(th, path, mode, x, images, monkeypatch, False)
    assert a.shape == b.shape and np.isfinite(b).all() and b.std() > 0
    if mode == 3:
        assert np.array_equal(a, b)
    else:
        assert np.abs(a - b).max() <= (2e-3 if mode == 1 else 1.6e-2) * np.abs(b).max()


@pytest.mark.parametrize("dtype", [K.THB_F32, K.THB_F16, K.THB_BF16, K.THB_U8])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("h,w,stride", [(6, 8, 24), (6, 8, 25), (6, 8, 30), (5, 7, 21), (5, 7, 22)])
def test_byte_pictures_at_any_address(dtype, offset, h, w, stride):
    """Space-to-depth of byte pictures through the kernel ABI, wherever they start and however long their rows are."""
    lib, (n, pad, mean, std) = K.load(), (2, 1, np.float32([0.45, 0.4, 0.5]), np.float32([0.225, 0.25, 0.2]))
    raw = np.random.default_rng(offset * 31 + w).integers(0, 256, 8 + n * h * stride, dtype=np.uint8)
    src = G.dev(raw)
    h2, w2 = (h + 1) // 2, (w + 1) // 2
    pitch = w2 + pad + 2
    outs = []
    for wrapper in ((False, True) if dtype in (K.THB_F16, K.THB_BF16) and not (h | w) & 1 else (False,)):
        y = torch.full((n, h2, pitch, 16), 77, dtype=G._TORCH[dtype], device="cuda")
        qs, qm = C.c_float(), C.c_float()
        at = C.c_void_p(src.data_ptr() + offset)
        st = (mean.ctypes.data_as(C.c_void_p), std.ctypes.data_as(C.c_void_p))
        if wrapper:
            rc = lib.thb_preprocess_images_s2d(at, n, h, w, stride, 0, *st, dtype, G.ptr(y), 16, pitch, pad, None)
        else:
            rc = lib.thb_preprocess_s2d_any(at, 1, None, n, 3, h, w, 2, stride, 0, *st, dtype, G.ptr(y), 16, pitch, pad, C.byref(qs),
                                            C.byref(qm), None)
        assert rc == 0
        outs.append(y.float().cpu().numpy())
    assert all(np.array_equal(o, outs[0]) for o in outs)
    img = np.lib.stride_tricks.as_strided(raw[offset:], (n, h, w, 3), (h * stride, stride, 3, 1))
    want = np.zeros((n, h2, pitch, 16), np.float32)
    if dtype == K.THB_U8:  # (the static range of the image loader)
        v = (0 - mean) / std
        zero = int(np.round(-np.float32(np.round(qs.value * np.float32(qm.value))))) & 255
        q = outs[0]
        assert np.array_equal(q[:, :, :pad], np.zeros_like(q[:, :, :pad])) and qs.value == v.min()
        sub = 255 * (mean + std * np.float32(qs.value))
        sub = np.sign(sub) * np.floor(np.abs(sub) + 0.5)
        val = np.floor((img - sub) * (np.float32(qm.value) / (255 * std)) + 0.5)
        full = np.full((n, 2 * h2, 2 * w2, 3), zero, np.float64)
    else:
        val = ((img.astype(np.float32) * np.float32(0.003921568)) - mean) * (np.float32(1) / std)
        full = np.zeros((n, 2 * h2, 2 * w2, 3), np.float32)
    full[:, :h, :w] = val
    for b in range(4):
        want[:, :, pad:pad + w2, 3 * b:3 * b + 3] = full[:, b >> 1::2, b & 1::2]
    assert np.abs(outs[0] - want).max() <= {K.THB_F32: 0, K.THB_F16: 2e-3, K.THB_BF16: 1.6e-2, K.THB_U8: 1}[dtype]
    assert (outs[0] != want).mean() <= (0 if dtype == K.THB_F32 else 0.02 if dtype == K.THB_U8 else 1)


def test_float_space_to_depth_entry_points():
    """the entry points for even sides and block size 2 agree with the general one"""
    lib, (n, h, w), mean, std = K.load(), (2, 6, 10), np.float32([0.45, 0.4, 0.5]), np.float32([0.225, 0.25, 0.2])
    x = G.dev(np.random.default_rng(5).standard_normal((n, 3, h, w)).astype(np.float32))
    st = (mean.ctypes.data_as(C.c_void_p), std.ctypes.data_as(C.c_void_p))
    for dtype, ld in ((K.THB_F32, 12), (K.THB_F16, 16), (K.THB_U8, 16)):
        a, b = (torch.full((n, h // 2, w // 2, ld), 7, dtype=G._TORCH[dtype], device="cuda") for _ in range(2))
        qs, qm = C.c_float(-4), C.c_float(20)
        assert lib.thb_preprocess_s2d_any(G.ptr(x), 0, None, n, 3, h, w, 2, 0, 0, *st, dtype, G.ptr(a), ld, w // 2, 0, C.byref(qs), C.byref(qm), None) == 0
        if dtype == K.THB_U8:
            assert lib.thb_preprocess_s2d_u8(G.ptr(x), None, n, 3, h, w, *st, G.ptr(b), ld, qs, qm, None) == 0
        else:
            assert lib.thb_preprocess_s2d(G.ptr(x), None, n, 3, h, w, *st, dtype, G.ptr(b), ld, None) == 0
        assert torch.equal(a, b) and a.float().std() > 0


@pytest.mark.parametrize("inplace", [False, True])
def test_float_space_to_depth_at_any_float_address(inplace):
    """planes that start at an odd float, whose pixel pairs are not 8-byte aligned, give what aligned ones give"""
    lib, (n, h, w), mean, std = K.load(), (2, 6, 10), np.float32([0.45, 0.4, 0.5]), np.float32([0.225, 0.25, 0.2])
    raw = np.random.default_rng(6).standard_normal(n * 3 * h * w).astype(np.float32)
    st = (mean.ctypes.data_as(C.c_void_p), std.ctypes.data_as(C.c_void_p))
    outs = []
    for lead in (0, 1):
        x = G.dev(np.concatenate([np.zeros(lead, np.float32), raw]))
        at = C.c_void_p(x.data_ptr() + 4 * lead)
        y = torch.full((n, h // 2, w // 2 + 3, 16), 7, dtype=torch.float16, device="cuda")
        assert lib.thb_preprocess_s2d_padded(at, at if inplace else None, n, 3, h, w, *st, K.THB_F16, G.ptr(y), 16, w // 2 + 3, 2, None) == 0
        outs.append((y.cpu(), x[lead:].cpu()))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert torch.equal(outs[0][1], torch.from_numpy(raw)) != inplace
    frame = torch.zeros(64, dtype=torch.uint8, device="cuda")
    assert lib.thb_preprocess_yuyv(C.c_void_p(frame.data_ptr() + 2), 2, 4, *st, K.THB_F16, G.ptr(y), 16, None) != 0
