"""The host side of a forward -- plans kept and dropped, sub-batches, where the uint8 input range comes from -- without a GPU: the
host library's own sources on a CUDA runtime and kernel launchers that compute nothing (fake_cuda.c).  Every test runs in a process
of its own, so that the fakes meet no other library."""
import os
import shutil
import subprocess
import sys

import pytest

from thnets_b200.capi import DEFAULT_LIB

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA", "/usr/local/cuda")

pytestmark = [
    pytest.mark.skipif(not os.path.exists(DEFAULT_LIB), reason="libthnets.so not built"),
    pytest.mark.skipif(shutil.which("gcc") is None or not os.path.exists(os.path.join(CUDA, "include")), reason="needs gcc and CUDA's headers"),
]


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    """Runs a test's code on the faked engine: `th` the binding, `lib` the library, `fake` its variables by name."""
    so = str(tmp_path_factory.mktemp("engine") / "libengine.so")
    csrc = os.path.join(ROOT, "thnets_b200", "csrc")
    host = [os.path.join(csrc, "host", f) for f in sorted(os.listdir(os.path.join(csrc, "host"))) if f.endswith(".c")]
    subprocess.check_call(["gcc", "-O1", "-w", "-std=gnu11", "-shared", "-fPIC", "-ffp-contract=off", "-fopenmp", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(csrc, "host"), "-I", os.path.join(csrc, "kernels"), "-I", os.path.join(CUDA, "include"), "-o", so]
                          + host + [os.path.join(ROOT, "tests", "fake_cuda.c"), DEFAULT_LIB, "-lm", "-Wl,-rpath," + os.path.dirname(DEFAULT_LIB)])
    head = f"""
import ctypes as C, os, sys
sys.path.insert(0, {ROOT!r})
os.environ["THB200_NO_EXIT"] = "1"
import numpy as np
from thnets_b200 import fixtures as fx
from thnets_b200.capi import THNets
th = THNets({so!r})
lib = th.lib
class Fake:
    kinds = dict(budget=C.c_size_t, live=C.c_size_t, q_sub=C.c_float, q_mult=C.c_float)
    def var(self, name):
        return self.kinds.get(name, C.c_int).in_dll(lib, "fake_" + name)
    def __getattr__(self, name):
        return self.var(name).value
    def __setattr__(self, name, v):
        self.var(name).value = v
fake = Fake()
def network(g, mode, path="net"):
    fx.write_pymodel(g, path)
    src = th.load_network(path)
    if mode == 3:
        net = th.create_lowp_network(src, 8.0)
    else:
        lib.THB200_SetPrecision(mode)
        net = lib.THCreateCudaNetwork(src)
    assert net
    th.free_network(src)
    return net
def pinned(shape):
    p = lib.THB200_HostAlloc(4 * int(np.prod(shape)))
    return np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), shape=shape)
def call(net, x, fn=None):
    res, ow, oh = C.POINTER(C.c_float)(), C.c_int(), C.c_int()
    n, c, h, w = x.shape
    return (fn or lib.THB200_ProcessFloatConst)(net, x.ctypes.data, n, w, h, c, C.byref(res), C.byref(ow), C.byref(oh))
"""

    def run(code, tmp_path, threads=4):
        env = dict(os.environ, OMP_NUM_THREADS=str(threads))
        r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, env=env, cwd=tmp_path)
        assert r.returncode == 0, r.stdout + r.stderr

    return run


@pytest.mark.parametrize("threads", [1, 4, 16])
@pytest.mark.parametrize("size", [64, 225])
def test_uint8_input_range(engine, tmp_path, threads, size):
    """A uint8 forward of a float batch takes its range from one pass: the host's staging of a pageable batch, a pass of the host's
    threads over a small page-locked one, the devices' pass over a large one -- and only there is the devices' pass launched, whatever
    the number of threads.  Where the host finds the range it is that of the normalised values, NaNs left out."""
    engine(f"""
size, threads = {size}, {threads}
g = fx.resnet18(width=0.25, size=size, classes=10, fc_bias=0.05)
net = network(g, 3)
mean, std = np.float32([0.45, 0.4, 0.5]), np.float32([0.225, 0.25, 0.2])
th.set_stats(net, mean, std)
def expected(x):
    v = (x - mean[None, :, None, None]) / std[None, :, None, None]
    lo, hi = min(0, np.nanmin(v)), max(0, np.nanmax(v))
    return np.float32(lo), np.float32(255.0 / float(hi - lo))
rng = np.random.default_rng(size)
for n in (1, 5, 67):
    for where in ("const", "inplace", "pinned"):
        x = (pinned if where == "pinned" else np.empty)((n, 3, size, size))
        x = x.astype(np.float32, copy=False)
        x[...] = rng.standard_normal(x.shape, dtype=np.float32)
        x[n // 2, 1, 7, 7:11] = np.nan
        x[n - 1, n % 3, size - 1, size - 1] = 9 + n  # the batch's very last values count
        x[0, 2, 0, 0] = -7 - n
        want, fake.minmax = expected(x), 0
        copy = x.copy()
        assert call(net, x, lib.THProcessFloat if where == "inplace" else None) > 0
        small = x.nbytes <= min(threads, 8) * 300 * 1024
        if where == "pinned" and not small:
            assert fake.minmax == 1, (n, where)
        else:
            assert fake.minmax == 0, (n, where)
            assert (np.float32(fake.q_sub), np.float32(fake.q_mult)) == want, (n, where, fake.q_sub, fake.q_mult, want)
        if where == "inplace":
            assert np.array_equal(x, (copy - mean[None, :, None, None]) / std[None, :, None, None], equal_nan=True)
        else:
            assert np.array_equal(x, copy, equal_nan=True)
assert fake.empty == 0
""", tmp_path, threads)


def test_sub_batches_make_room(engine, tmp_path):
    """A shape whose sub-batch plans do not fit beside the plans of earlier shapes makes those give way, as a shape's own plan does;
    when nothing is left to give way the call fails and a smaller one still works."""
    engine("""
g = fx.resnet18(width=0.25, size=64, classes=10)
x = {n: pinned((n, 3, 64, 64)) for n in (1, 8, 16)}
def sizes():
    net = network(g, 1)
    lib.THB200_SetPipelineChunks(1)
    assert call(net, x[8]) > 0
    whole = fake.live
    lib.THB200_SetPipelineChunks(2)
    assert call(net, x[8]) > 0
    both = fake.live
    th.free_network(net)
    assert fake.live == 0
    return whole, both
whole, both = sizes()
net = network(g, 1)
lib.THB200_SetPipelineChunks(1)
assert call(net, x[16]) > 0
assert call(net, x[1]) > 0
fake.budget = fake.live + whole // 2 + (both - whole) // 2
assert both <= fake.budget
lib.THB200_SetPipelineChunks(2)
for _ in range(3):
    assert call(net, x[8]) > 0, lib.THB200_LastErrorString()
assert fake.live >= both
fake.budget = 1000
assert call(net, x[16]) <= 0
fake.budget = 1 << 50
assert call(net, x[16]) > 0
""", tmp_path)


def test_plan_memory_bound(engine, tmp_path):
    """The plans an engine keeps stay within their bound in bytes, their sub-batches included, the one in use is never dropped, and
    dropped shapes are planned again."""
    engine("""
LIMIT = 12 << 30
net = network(fx.segnet(), 1)
lib.THB200_SetPipelineChunks(2)
x = pinned((23, 3, 512, 512))
assert call(net, x[:1]) > 0
weights = fake.live  # (an upper bound: with the smallest plan)
seen = set()
for n in (20, 21, 22, 23, 20, 1, 22):
    before = fake.live
    assert call(net, x[:n]) > 0, lib.THB200_LastErrorString()
    assert fake.live <= LIMIT + weights, (n, fake.live / 2**30)
    seen.add(fake.live < before)
assert fake.live > LIMIT // 4 and len(seen) == 2, "some plans were kept and some dropped"
th.free_network(net)
assert fake.live == 0
""", tmp_path)


def test_a_plan_that_does_not_fit_leaves_nothing_behind(engine, tmp_path):
    """whatever allocation a plan fails at, its streams and memory are given back"""
    engine("""
g = fx.resnet18(width=0.25, size=64, classes=10)
net = network(g, 1)
x = pinned((8, 3, 64, 64))
assert call(net, x[:1]) > 0
for room in (0, 8, 64, 1 << 10, 1 << 17, 1 << 18, 1 << 20):
    th.free_network(net)
    assert fake.streams == 0 and fake.live == 0
    net = network(g, 1)
    fake.budget = room
    assert call(net, x) <= 0
    assert fake.streams == 0, room
    fake.budget = 1 << 50
""", tmp_path)


def test_no_empty_sub_batch(engine, tmp_path):
    """Every sub-batch of every GPU's slice has an image, whether the engine cuts the batch by its model or on request, and all of
    the images are computed.  (The network's first launch is none that could start on a part of the batch, so that the model cuts.)"""
    engine("""
fake.devices = 2
cut = 0
for gpus in (1, 2):
    lib.THB200_SetDevices(gpus)
    for side in (512, 1024, 2048):
        g = fx.Graph()
        t = g.conv(g.relu(g.conv(g.bn(0, 3), 3, 64, 3, pad=1)), 64, 64, 3, pad=1)
        g.linear(g.view(g.avgpool(t, side), 64), 64, 5)
        net = network(g, 1)
        x = pinned((17, 3, side, side))
        for chunks in (0, 2, 3, 4):
            lib.THB200_SetPipelineChunks(chunks)
            for n in range(2, 18):
                fake.boundaries = fake.images = 0
                assert call(net, x[:n]) > 0
                assert fake.empty == 0, (gpus, side, chunks, n)
                assert fake.images == n
                cut += chunks == 0 and fake.boundaries > gpus
        th.free_network(net)
assert cut > 40, "the model cut some of the batches"
""", tmp_path)


def test_sliced_start_of_a_batch_normalised_in_place(engine, tmp_path):
    """a large page-locked batch starts part by part whether or not its normalised values go back to the caller"""
    engine("""
net = network(fx.resnet18(size=224, classes=10), 1)
th.set_stats(net, (0.45,) * 3, (0.225,) * 3)
x = pinned((67, 3, 224, 224))
lib.THB200_SetPipelineChunks(1)
parts = []
for fn in (lib.THB200_ProcessFloatConst, lib.THProcessFloat):
    fake.boundaries = fake.images = 0
    assert call(net, x, fn) > 0
    assert fake.images == 67
    parts.append(fake.boundaries)
assert parts[0] == parts[1] > 1, parts
""", tmp_path)


def test_split_weights_make_room(engine, tmp_path):
    """The second copies of fp32 weights never cost a call its memory: where a plan, or its sub-batches, fit without them only, they go
    and the convolutions run on the FP32 units; a smaller shape gets them back.  THB200_NO_F32_TC=1 does without them from the start."""
    engine("""
fake.f32_tc = 1
g = fx.resnet18(width=0.5, size=64, classes=10)
x = pinned((64, 3, 64, 64))
def held(chunks, env=None):
    if env:
        os.environ["THB200_NO_F32_TC"] = env
    lib.THB200_SetPipelineChunks(chunks)
    net = network(g, 0)
    fake.splits = fake.tc_launches = 0
    assert call(net, x) > 0
    live = fake.live
    assert (fake.splits > 0) == (fake.tc_launches > 0) == (env != "1")
    th.free_network(net)
    assert fake.live == 0
    os.environ.pop("THB200_NO_F32_TC", None)
    return live
for chunks in (1, 2):
    without, full = held(chunks, "1"), held(chunks, "0")
    assert full > 1.1 * without
    for part in (0.0, 0.02, 0.2, 0.5, 0.9, 0.999, 1.0):
        net = network(g, 0)
        fake.budget = without + int(part * (full - without))
        fake.tc_launches = 0
        for _ in range(2):
            assert call(net, x) > 0, (chunks, part, lib.THB200_LastErrorString())
        assert fake.live <= fake.budget and (part < 1 or fake.tc_launches > 0)
        fake.budget = 1 << 50
        fake.tc_launches = 0
        assert call(net, x[:3]) > 0 and fake.tc_launches > 0, "a shape planned later has them again"
        assert call(net, x) > 0
        th.free_network(net)
        assert fake.live == 0 and fake.streams == 0
    net = network(g, 0)
    fake.budget = without - (1 << 20)
    assert call(net, x) <= 0
    fake.budget = 1 << 50
    assert call(net, x) > 0
    th.free_network(net)
""", tmp_path)


def test_one_wait_a_plan(engine, tmp_path):
    """What a plan launches to lay its weights out is waited for once, however many layers it has."""
    engine("""
fake.f32_tc = 1
net = network(fx.resnet18(width=0.5, size=64, classes=10), 0)
x = pinned((8, 3, 64, 64))
lib.THB200_SetPipelineChunks(1)
for n in (1, 2, 8):
    fake.waits = 0
    assert call(net, x[:n]) > 0
    assert fake.waits == 1
    assert call(net, x[:n]) > 0
    assert fake.waits == 1
assert fake.splits > 10
""", tmp_path)
