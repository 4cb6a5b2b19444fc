"""A large batch whose first launches follow its copy to the GPU part by part: bit for bit the result of the same batch sent
whole."""
import os

import numpy as np
import pytest

from thnets_b200 import fixtures as fx
from thnets_b200.capi import THNets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def th():
    return THNets()


def run(th, path, mode, batch, images, slices):
    os.environ["THB200_NO_SLICES"] = "0" if slices else "1"
    try:
        h = th.load_network(path)
        th.set_stats(h, (0.45,) * 3, (0.225,) * 3)
        if mode == 3:
            net = th.create_lowp_network(h, 8.0)
        else:
            th.lib.THB200_SetPrecision(mode)
            net = th.lib.THCreateCudaNetwork(h)
            th.lib.THB200_SetPrecision(0)
        assert net
        th.free_network(h)
        th.lib.THB200_SetPipelineChunks(1)
        outs = [(th.process_images(net, batch) if images else th.process_float(net, batch))[0] for _ in range(3)]
        th.free_network(net)
    finally:
        th.lib.THB200_SetPipelineChunks(0)
        os.environ.pop("THB200_NO_SLICES")
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    return outs[0]


@pytest.mark.parametrize("mode", [0, 1, 3], ids=["fp32", "fp16", "uint8"])
@pytest.mark.parametrize("images", [True, False], ids=["bytes", "floats"])
@pytest.mark.parametrize("net,batch,size", [("resnet18", 67, 224), ("resnet50", 129, 160), ("resnet18", 61, 225)])
def test_sliced_start(th, tmp_path, mode, images, net, batch, size):
    if mode == 3 and not images:
        pytest.skip("the uint8 engine measures a float batch before it starts")
    g = getattr(fx, net)(width=0.25 if mode == 0 else 1.0, size=size, classes=10, fc_bias=0.05)
    path = str(tmp_path / "n.net")
    fx.write_pymodel(g, path)
    rng = np.random.default_rng(batch)
    if images:
        x = [rng.integers(0, 256, (size, size, 3), dtype=np.uint8) for _ in range(batch)]
    else:
        x = rng.standard_normal((batch, 3, size, size), dtype=np.float32)
    assert np.array_equal(run(th, path, mode, x, images, True), run(th, path, mode, x, images, False))
