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


@pytest.mark.parametrize("mode", [0, 1], ids=["fp32", "fp16"])
def test_sliced_start_in_place(th, tmp_path, monkeypatch, mode):
    """A page-locked float batch that is normalised in place: sliced or whole, the same scores, and in the caller's buffer exactly
    the normalised values."""
    import ctypes
    batch, size, mean, std = 67, 225, np.float32([0.45, 0.4, 0.5]), np.float32([0.225, 0.25, 0.2])
    path = str(tmp_path / "n.net")
    fx.write_pymodel(fx.resnet18(width=0.25 if mode == 0 else 1.0, size=size, classes=10, fc_bias=0.05), path)
    x = np.random.default_rng(3).standard_normal((batch, 3, size, size), dtype=np.float32)
    p = th.lib.THB200_HostAlloc(x.nbytes)
    pinned = np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), shape=x.shape)
    th.lib.THB200_SetPipelineChunks(1)
    outs = []
    try:
        for off in ("0", "1"):
            monkeypatch.setenv("THB200_NO_SLICES", off)
            h = th.load_network(path)
            th.set_stats(h, mean, std)
            th.lib.THB200_SetPrecision(mode)
            net = th.lib.THCreateCudaNetwork(h)
            th.lib.THB200_SetPrecision(0)
            th.free_network(h)
            for _ in range(3):
                pinned[...] = x
                outs.append(th.process_float(net, pinned, copy_input=False)[0])
                assert np.array_equal(pinned, (x - mean[:, None, None]) / std[:, None, None])
            th.free_network(net)
    finally:
        th.lib.THB200_SetPipelineChunks(0)
        th.lib.THB200_HostFree(p)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])


@pytest.mark.parametrize("net,batch,size", [("resnet18", 5, 97), ("resnet18", 66, 224), ("vgg16", 40, 224)])
@pytest.mark.parametrize("nan", [False, True], ids=["finite", "nan"])
def test_uint8_range_found_by_the_host(th, tmp_path, net, batch, size, nan):
    """A uint8 forward of a float batch with the range found wherever it is found -- by the host's threads while they stage a
    pageable batch, as it is or normalising it in place, by a pass of theirs over a small page-locked one, by the device's pass
    over a large one -- and with many threads or few: the same bytes."""
    import ctypes
    omp = ctypes.CDLL("libgomp.so.1")
    threads_before = omp.omp_get_max_threads()
    g = fx.vgg16(width=0.25, classes=10, fc=64) if net == "vgg16" else fx.resnet18(width=0.25, size=size, classes=10, fc_bias=0.05)
    path = str(tmp_path / "n.net")
    fx.write_pymodel(g, path)
    x = np.random.default_rng(batch).standard_normal((batch, 3, size, size), dtype=np.float32)
    if nan:
        x[batch // 2, 1, 7, 7:11] = np.nan
    p = th.lib.THB200_HostAlloc(x.nbytes)
    pinned = np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), shape=x.shape)
    pinned[...] = x
    outs = []
    for threads in (8, 2):
        omp.omp_set_num_threads(threads)
        try:
            h = th.load_network(path)
            th.set_stats(h, (0.45, 0.4, 0.5), (0.225, 0.25, 0.2))
            net_h = th.create_lowp_network(h, 8.0)
            th.free_network(h)
            outs += [th.process_float(net_h, b)[0] for b in (x, x, pinned, x, pinned)]
            outs.append(th.process_float(net_h, x.copy(), copy_input=False)[0])
            th.free_network(net_h)
        finally:
            omp.omp_set_num_threads(threads_before)
    th.lib.THB200_HostFree(p)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])
