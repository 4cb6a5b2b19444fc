"""First convolutions of stride 2 and 4 on a space-to-depth input (any side lengths, floats and byte pictures, one picture or
a batch) against the same network with the layer as it is: uint8 bit for bit, 16-bit types up to the order of the sums."""
import numpy as np
import pytest

from thnets_b200 import fixtures as fx
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
