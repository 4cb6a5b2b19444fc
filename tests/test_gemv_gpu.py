"""Linear on up to eight rows: every count of rows of x, weight rows that do not divide among the CTAs or their groups of four or two, and
reductions of less than, exactly and just over whole batches of 256 vectors."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from thnets_b200 import kernels_abi as K

pytestmark = pytest.mark.gpu

UNIT = {K.THB_F32: 2.0 ** -24, K.THB_F16: 2.0 ** -11, K.THB_BF16: 2.0 ** -8}
TORCH = {K.THB_F32: torch.float32, K.THB_F16: torch.float16, K.THB_BF16: torch.bfloat16}


@pytest.fixture(scope="module")
def lib():
    return K.load()


@pytest.mark.parametrize("dtype", [K.THB_F32, K.THB_F16, K.THB_BF16])
@pytest.mark.parametrize("m,vectors", [(1, 1), (5, 255), (296, 256), (593, 257), (1000, 512), (1187, 3), (4096, 769), (592, 1025), (1184, 513)])
def test_gemv_edges(lib, dtype, m, vectors):
    per = 4 if dtype == K.THB_F32 else 8
    k, td = vectors * per, TORCH[dtype]
    g = torch.Generator(device="cuda").manual_seed(m)
    w = torch.randn(m, k, device="cuda", generator=g).to(td)
    yld = (m + per - 1) // per * per + per
    for n in range(1, 9):
        x = torch.randn(n, k + per, device="cuda", generator=g).to(td)  # a pitch beyond K
        shift = torch.randn(m, device="cuda", generator=g)
        y = torch.full((n, yld), 7.0, device="cuda", dtype=td)
        rc = lib.thb_gemv_fwd(dtype, x.data_ptr(), n, k, k + per, w.data_ptr(), m, None, shift.data_ptr(), None, y.data_ptr(), yld, None)
        torch.cuda.synchronize()
        assert rc == 0
        xd = x[:, :k].double()
        ref = xd @ w.double().T + shift.double()
        # the products' rounding errors in fp32 (a thread adds at most K / 256 + one vector in a row, then thirteen more sums), and
        # one rounding to the result's type
        bound = (k / 256 + per + 14) * 2.0 ** -24 * (xd.abs() @ w.double().abs().T + shift.double().abs()) + UNIT[dtype] * ref.abs() + 1e-30
        assert bool(((y[:, :m].double() - ref).abs() <= bound).all())
        pad = (m + per - 1) // per * per
        assert bool((y[:, m:pad] == 0).all()) and bool((y[:, pad:] == 7).all())
