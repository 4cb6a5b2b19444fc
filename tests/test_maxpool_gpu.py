"""Max pooling by vectors: windows of 2 x 2 and 3 x 3 with any stride and padding, edges of the rows a block takes, and in uint8
the pixel sums it leaves, against numpy."""
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
    lib.thb_maxpool_sums.argtypes = [C.c_int, C.c_void_p] + [C.c_int] * 13 + [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    return lib


def pooled(x, k, s, p, oh, ow, start):
    n, c, h, w = x.shape
    y = np.full((n, c, oh, ow), start, x.dtype)
    for r in range(k):
        for q in range(k):
            for i in range(oh):
                for j in range(ow):
                    a, b = i * s - p + r, j * s - p + q
                    if 0 <= a < h and 0 <= b < w:
                        v = x[:, :, a, b]
                        y[:, :, i, j] = np.where(v > y[:, :, i, j], v, y[:, :, i, j])
    return y


CASES = [  # n, c, h, w, k, stride, pad, output rows and columns
    (2, 64, 12, 14, 2, 2, 0, 6, 7),
    (1, 16, 9, 300, 2, 1, 1, 10, 301),   # rows of more than one block, one group of channels
    (3, 20, 7, 7, 3, 1, 1, 7, 7),
    (1, 512, 6, 5, 2, 2, 0, 3, 3),       # 32 groups; the last column's window is half outside
    (2, 256, 13, 11, 3, 2, 0, 6, 5),
    (2, 33, 10, 10, 3, 3, 1, 4, 4),      # three groups: no sums
    (2, 64, 11, 9, 3, 2, 1, 6, 5),       # 3x3 stride 2: two rows of outputs a thread (16-bit types), the last
    (1, 32, 14, 6, 3, 2, 0, 7, 3),       # thread's second one inside, or beyond the output
    (300, 16, 23, 7, 3, 2, 0, 11, 3),    # in uint8 from this many blocks on
    (1, 3, 1, 1, 2, 2, 0, 1, 1),
]


@pytest.mark.parametrize("dtype", [K.THB_F32, K.THB_F16, K.THB_BF16, K.THB_U8], ids=["fp32", "fp16", "bf16", "uint8"])
@pytest.mark.parametrize("case", CASES)
def test_vectors(lib, case, dtype):
    n, c, h, w, k, s, p, oh, ow = case
    rng = np.random.default_rng(c)
    if dtype == K.THB_U8:
        x = rng.integers(0, 256, (n, c, h, w)).astype(np.uint8)
    else:
        x = rng.standard_normal((n, c, h, w)).astype(np.float32)
        x[0, 0, 0, 0], x[-1, -1, -1, -1] = np.nan, -np.inf
        x = torch.from_numpy(x).to(G._TORCH[dtype]).float().numpy()
    lowest = 0 if dtype == K.THB_U8 else -np.finfo(np.float32).max if dtype == K.THB_F32 else -np.inf
    ref = pooled(x, k, s, p, oh, ow, lowest)
    xt, ld = G.to_nhwc(x, dtype)
    y = torch.full((n, oh, ow, ld + K.ALIGN[dtype]), 7, dtype=xt.dtype, device="cuda")
    assert lib.thb_maxpool(dtype, G.ptr(xt), n, h, w, c, ld, k, k, s, s, p, p, oh, ow, G.ptr(y), y.shape[-1], None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(G.from_nhwc(y, c), ref) and bool((y[..., ld:] == 7).all())
    if dtype != K.THB_U8:
        return
    sums = torch.full((n * oh * ow + 1,), -5, dtype=torch.int32, device="cuda")
    y2 = torch.zeros_like(y)
    rc = lib.thb_maxpool_sums(dtype, G.ptr(xt), n, h, w, c, ld, k, k, s, s, p, p, oh, ow, G.ptr(y2), y.shape[-1], G.ptr(sums), None)
    torch.cuda.synchronize()
    groups = (c + 15) // 16
    if groups & (groups - 1):
        assert rc != 0
        return
    assert rc == 0 and np.array_equal(G.from_nhwc(y2, c), ref)
    assert np.array_equal(sums[:-1].cpu().numpy(), ref.astype(np.int64).sum(1).ravel()) and int(sums[-1]) == -5
