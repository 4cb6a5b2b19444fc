"""Plans kept per input shape: a network that comes back to a shape it used before, or that meets more shapes than are
kept, computes what a freshly converted network computes."""
import numpy as np
import pytest

from thnets_b200 import fixtures as fx
from thnets_b200.capi import THNets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def th():
    return THNets()


def convert(th, path, mode):
    h = th.load_network(path)
    if mode == 3:
        net = th.create_lowp_network(h, 8.0)
    else:
        th.lib.THB200_SetPrecision(mode)
        net = th.lib.THCreateCudaNetwork(h)
        th.lib.THB200_SetPrecision(0)
    assert net, th.lib.THB200_LastErrorString()
    th.free_network(h)
    return net


@pytest.mark.parametrize("mode", [0, 1, 3], ids=["fp32", "fp16", "uint8"])
def test_shapes_in_turn(th, tmp_path, mode):
    g = fx.resnet18(width=0.25, size=64, classes=10, fc_bias=0.05)
    path = str(tmp_path / "r.net")
    fx.write_pymodel(g, path)
    net = convert(th, path, mode)
    batches = (5, 2, 7, 1, 3, 9, 5, 1, 2, 9)  # six shapes, more than are kept; the later ones return to earlier ones
    want = {}
    for n in sorted(set(batches)):
        fresh = convert(th, path, mode)
        want[n] = th.process_float(fresh, g.make_input(n, seed=n))[0]
        th.free_network(fresh)
    for n in batches:
        for _ in range(3):  # launched directly, captured, replayed
            out, _, _ = th.process_float(net, g.make_input(n, seed=n))
            assert np.array_equal(out, want[n])
    th.free_network(net)
