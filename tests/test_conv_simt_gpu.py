"""The fp32 convolution at the edges of its tiles (64 and 128 pixels and channels, K blocks of 32), in every split of its
reduction, against a double-precision convolution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import torch  # noqa: E402

from thnets_b200 import kernels_abi as K  # noqa: E402
from tests import gpu_util as G  # noqa: E402


@pytest.fixture(scope="module")
def lib():
    return K.load()


CASES = [  # n, cin, h, w, cout, k, stride, pad
    (1, 8, 7, 9, 128, 3, 1, 1),       # 63 pixels, K = 72
    (1, 36, 8, 8, 64, 3, 1, 1),       # 64 pixels
    (1, 128, 5, 13, 130, 3, 1, 1),    # 65 pixels, channels beyond a tile
    (1, 100, 127, 1, 256, 1, 1, 0),   # 127 pixels, K = 100
    (3, 64, 9, 5, 200, 3, 2, 1),
    (1, 3, 43, 3, 72, 1, 1, 0),       # 129 pixels, one K block
    (2, 64, 40, 41, 128, 3, 1, 1),
    (70, 16, 20, 20, 128, 1, 1, 0),   # unsplit, wide tiles
]


@pytest.mark.parametrize("case", CASES)
def test_tiles_and_splits(lib, case):
    n, cin, h, w, cout, k, s, p = case
    rng = np.random.default_rng(cin)
    x = rng.standard_normal((n, cin, h, w)).astype(np.float32)
    wt = (rng.standard_normal((cout, cin, k, k)) * (cin * k * k) ** -0.5).astype(np.float32)
    shift = rng.standard_normal(cout).astype(np.float32)
    ref = torch.nn.functional.conv2d(torch.from_numpy(x).double().cuda(), torch.from_numpy(wt).double().cuda(), stride=s,
                                     padding=p).cpu().numpy() + shift[None, :, None, None]
    res = rng.standard_normal(ref.shape).astype(np.float32)
    ref = np.maximum(ref - res, 0)
    xt, _ = G.to_nhwc(x, K.THB_F32)
    for splits in (0, 1, 2, 4, 8, 16):
        conv = G.Conv(lib, K.THB_F32, x.shape, wt, (s, s), (p, p))
        conv.set_affine(None, shift)
        rt, rld = G.to_nhwc(res, K.THB_F32)
        conv.set_residual(rt, rld, 1.0, -1.0)
        conv.set_act(K.ACT_THRESHOLD)
        conv.d.splits = splits
        out_ld = G.ru(cout, 4) + 4
        y = conv.run(xt, out_ld=out_ld, fill=3.0)
        assert bool((y[..., out_ld - 4:] == 3.0).all()), "wrote beyond its channels"
        out = G.from_nhwc(y, cout)
        assert G.rel_err(out, ref) < 2e-6, splits
        assert np.array_equal(out, G.from_nhwc(conv.run(xt), cout)), splits
