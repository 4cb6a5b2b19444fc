"""The cache of TMA descriptors behind the tensor-core convolutions: full, and shared by host threads."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from thnets_b200 import kernels_abi as K  # noqa: E402
from tests import gpu_util as G  # noqa: E402


@pytest.fixture(scope="module")
def lib():
    return K.load()


@pytest.mark.parametrize("cout", [64, 256])
def test_more_descriptors_than_the_cache_holds(lib, cout, monkeypatch):
    """Each launch finds the descriptors of its activations and its output and needs a new one for its residual, which takes the place of
    every other one in turn, those of the same launch among them."""
    rng = np.random.default_rng(cout)
    n, side = 1100, 40
    x = rng.standard_normal((1, 64, side, side)).astype(np.float32)
    conv = G.Conv(lib, K.THB_F16, x.shape, rng.standard_normal((cout, 64, 1, 1)).astype(np.float32) / 8)
    xt, conv.d.in_ld = G.to_nhwc(x, K.THB_F16)
    monkeypatch.setenv("THB200_FEW_TILES", "0")  # the persistent kernel: it has a descriptor for each of its tensors
    lib.thb_conv_reload_knobs()
    plain = conv.run(xt)
    res = torch.arange(n, device="cuda").half().view(n, 1, 1, 1).expand(n, side, side, cout).contiguous()
    y = torch.zeros((1, side, side, cout), dtype=torch.half, device="cuda")
    conv.d.res_ld, conv.d.self_coef, conv.d.res_coef = cout, 0.0, 1.0
    wrong = torch.zeros(1, dtype=torch.int64, device="cuda")
    for i in range(n):
        conv.d.self_coef = 1.0 if i % 2 else 0.0
        conv.d.res = res[i].data_ptr()
        assert lib.thb_conv_fwd(C.byref(conv.d), G.ptr(xt), G.ptr(y), None) == 0
        want = (plain.float() * conv.d.self_coef + i).half()
        wrong += ((y.float() - want.float()).abs() > 1e-3 * (i + 4)).sum()
    monkeypatch.undo()
    lib.thb_conv_reload_knobs()
    assert int(wrong) == 0 and bool((res == torch.arange(n, device="cuda").half().view(n, 1, 1, 1)).all())


def test_threads(lib):
    """Four host threads on streams of their own, fp32 and fp16 convolutions of hundreds of buffers: every result is its own input's."""
    rng = np.random.default_rng(1)
    wt = (rng.standard_normal((64, 64, 3, 3)) / 24).astype(np.float32)
    errors = []

    def work(t):
        dtype = K.THB_F32 if t % 2 else K.THB_F16
        conv = G.Conv(lib, dtype, (1, 64, 8, 8), wt, (1, 1), (1, 1))
        d = conv.d
        x = torch.randn(300, 8, 8, 64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(t)).to(G._TORCH[dtype])
        y = torch.zeros_like(x)
        ref = torch.nn.functional.conv2d(x.permute(0, 3, 1, 2).double(), torch.from_numpy(wt).to(G._TORCH[dtype]).cuda().double(), padding=1).permute(0, 2, 3, 1)
        parts = G.dzeros(lib.thb_conv_f32_split_bytes(C.byref(d))) if dtype == K.THB_F32 else None
        if parts is not None:
            assert lib.thb_conv_f32_split_weights(C.byref(d), parts.data_ptr(), None) == 0
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        for i in range(300):
            args = (x[i].data_ptr(), y[i].data_ptr(), C.c_void_p(stream.cuda_stream))
            rc = lib.thb_conv_f32_fwd(C.byref(d), parts.data_ptr(), *args) if parts is not None else lib.thb_conv_fwd(C.byref(d), *args)
            if rc:
                errors.append((t, i, rc))
        stream.synchronize()
        off = (y.double() - ref).abs().amax(dim=(1, 2, 3))
        errors.extend((t, int(i)) for i in torch.nonzero(off > (1e-5 if dtype == K.THB_F32 else 1e-2)).flatten()[:3])

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
