"""The forward passes that a program built on this framework spends its time in, as measurable cases.

Every case is one use of the public API on data in host memory, as the API takes it: a network is loaded and converted
once, then `THProcessFloat` / `THProcessImages` is called on batches.  A pass is the whole call: the copy of the batch
to the GPU, the forward, the copy of the result back.  Networks and precisions are the repository's own benchmark
architectures (thnets_b200/fixtures.py) with their seeded weights; inputs are made from the case's seed.

Fields of a case:
  net      resnet18 | resnet50 | vgg16 | alexnet_owt | segnet
  mode     fp32 | fp16 | bf16 | int8 (the uint8 "lowp" engine)
  batch    images of one call; last > 0: `calls` calls of `batch` images and one of `last`
  height, width   of the images
  source   images: byte pictures, each in an array of its own, as a decoder or a camera leaves them
           array:  a float batch in ordinary memory through the Python wrapper
           pinned: a float batch in memory from THB200_HostAlloc, the call made as a C program makes it
"""
from __future__ import annotations

import collections
import ctypes as C
import functools
import os
import tempfile
import weakref

import numpy as np
import torch

os.environ.setdefault("THB200_NO_EXIT", "1")  # a failing call raises here instead of ending the process

from thnets_b200 import fixtures as fx  # noqa: E402
from thnets_b200.capi import THNets  # noqa: E402

RANGE = 20.0                # output range of the uint8 engine, as the benchmark converts its networks
STATS = (0.45, 0.225)       # mean and deviation of byte pictures scaled to [0, 1)
MODES = {"fp32": 0, "fp16": 1, "bf16": 2}
WEIGHT_BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "int8": 1}
LARGEST_FLOPS = 2.2e12      # no drawn case computes more than ResNet-50 on 256 images


def _case(name, net, mode, batch, height, width, source, calls=1, last=0, spatial=False):
    return dict(name=name, net=net, mode=mode, batch=batch, height=height, width=width, source=source, calls=calls,
                last=last, spatial=spatial)


def listed():
    return [
        # one picture at a time, full precision: the reference's own command-line use, latency of a single small call
        _case("alexnet_fp32_1", "alexnet_owt", "fp32", 1, 224, 224, "array"),
        # a camera frame at a time through a small and a large classifier in half precision
        _case("resnet18_fp16_1", "resnet18", "fp16", 1, 224, 224, "images"),
        _case("resnet50_fp16_8", "resnet50", "fp16", 8, 224, 224, "images"),
        # a service's small batch in full precision, pictures of an odd size
        _case("resnet18_fp32_9_odd", "resnet18", "fp32", 9, 225, 225, "array"),
        # a classifier slid over a whole video frame (THMakeSpatial)
        _case("alexnet_fp16_frame", "alexnet_owt", "fp16", 1, 480, 640, "images", spatial=True),
        # one street scene through the segmentation network, neither side a power of two
        _case("segnet_bf16_1", "segnet", "bf16", 1, 368, 496, "pinned"),
        # the ordinary training-set-sized batches of the benchmark configurations
        _case("resnet18_fp16_64", "resnet18", "fp16", 64, 224, 224, "pinned"),
        _case("vgg16_int8_32", "vgg16", "int8", 32, 224, 224, "pinned"),
        _case("segnet_fp16_16", "segnet", "fp16", 16, 512, 512, "pinned"),
        # a directory of pictures in batches, the last one short
        _case("resnet18_bf16_ragged", "resnet18", "bf16", 64, 224, 224, "images", calls=2, last=37),
        # the headline configuration in both tensor-core precisions, fed with pictures
        _case("resnet50_fp16_256", "resnet50", "fp16", 256, 224, 224, "images"),
        _case("resnet50_int8_256", "resnet50", "int8", 256, 224, 224, "images"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("classify", "classify", "classify", "floats", "frame", "segment", "ragged"))
    if kind in ("classify", "floats"):
        net = rng.choice(("resnet18", "resnet50", "vgg16") if kind == "floats" else ("resnet18", "resnet50"))
        modes = {"vgg16": ("fp16", "int8")}.get(net, ("fp16", "bf16", "int8") + (("fp32",) if kind == "floats" else ()))
        mode = rng.choice(modes)
        side = 224 if net == "vgg16" or rng.random() < 0.5 else rng.randint(161, 320)
        # full precision runs on the FP32 units: batches as a service has them, not the benchmark's
        most = {"fp32": 16}.get(mode, {"vgg16": 48, "resnet50": 256, "resnet18": 256}[net])
        source = "images" if kind == "classify" else rng.choice(("array", "pinned"))
        c = _case("", net, mode, _log_int(rng, 1, min(most, 128) if kind == "floats" else most), side, side, source)
    elif kind == "frame":
        c = _case("", "alexnet_owt", rng.choice(("fp16", "bf16", "fp32")), 1, rng.randint(240, 720), rng.randint(320, 960),
                  "images", spatial=True)
    elif kind == "segment":
        c = _case("", "segnet", rng.choice(("fp16", "bf16")), _log_int(rng, 1, 16), 16 * rng.randint(12, 32),
                  16 * rng.randint(12, 32), "pinned")
    else:
        batch = _log_int(rng, 16, 128)
        c = _case("", "resnet18", rng.choice(("fp16", "bf16")), batch, 224, 224, "images", calls=rng.randint(1, 2),
                  last=rng.randint(1, batch - 1))
    one = _flops(c["net"], c["height"], c["width"], c["spatial"])
    c["batch"] = max(1, min(c["batch"], int(LARGEST_FLOPS / one)))
    del c["name"]
    return c


# ---- the network of a case -------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _graph(net, mode, height, width):
    build = getattr(fx, net)
    if net in ("resnet18", "resnet50"):
        # the uint8 engine cannot quantise an all-zero bias
        return build(size=height, fc_bias=0.01 if mode == "int8" else "zero")
    return build()  # vgg16 and alexnet_owt are trained at 224; segnet takes any size


@functools.lru_cache(maxsize=1)
def _lib():
    return THNets()


class _Net:
    """A converted network, freed with the last state that holds it."""

    def __init__(self, net, mode, height, width, source, spatial):
        th, g = _lib(), _graph(net, mode, height, width)
        self.th = th
        with tempfile.TemporaryDirectory() as tmp:
            path = os.path.join(tmp, net)
            if g.is_sequential():
                fx.write_torch7(g, path)
            else:
                fx.write_pymodel(g, path)
            src = th.load_network(path)
        if net == "vgg16" and mode == "int8":
            th.make_spatial(src, 224)  # the uint8 engine's classifier layers are convolutions, as the benchmark has them
        elif spatial:
            th.make_spatial(src, 224)
        if source == "images":
            th.set_stats(src, (STATS[0],) * 3, (STATS[1],) * 3)
        if mode == "int8":
            self.handle = th.create_lowp_network(src, RANGE)
        else:
            th.lib.THB200_SetPrecision(MODES[mode])
            self.handle = th.lib.THCreateCudaNetwork(src)
            th.lib.THB200_SetPrecision(0)
            if not self.handle:
                raise RuntimeError("THCreateCudaNetwork returned NULL")
        th.free_network(src)
        weakref.finalize(self, th.free_network, self.handle)


_nets = collections.OrderedDict()  # the last two: a program converts a network once and calls it on many batches


def _net_of(case):
    resnet = case["net"] in ("resnet18", "resnet50")
    key = (case["net"], case["mode"], case["height"] if resnet else 0, case["width"] if resnet else 0,
           "images" if case["source"] == "images" else "floats", case["spatial"])
    if key not in _nets:
        while len(_nets) > 1:
            _nets.popitem(last=False)
        _nets[key] = _Net(*key)
    _nets.move_to_end(key)
    return _nets[key]


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _pinned(th, shape):
    nbytes = 4 * int(np.prod(shape))
    p = th.lib.THB200_HostAlloc(nbytes)
    if not p:
        raise MemoryError("THB200_HostAlloc of %d bytes" % nbytes)
    a = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), shape=shape)
    return a, p


def _pictures(n, h, w, gen):
    """Byte pictures [n, h, w, 3]: large smooth areas with texture on them."""
    coarse = torch.rand((n, 3, 1 + h // 32, 1 + w // 32), generator=gen, device="cuda")
    img = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=True)
    img += 0.05 * torch.randn((n, 3, h, w), generator=gen, device="cuda")
    return img.mul_(255).clamp_(0, 255).to(torch.uint8).permute(0, 2, 3, 1).contiguous().cpu().numpy()


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.net = case, _net_of(case)
    th = s.net.th
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w = case["batch"], case["height"], case["width"]
    if case["source"] == "images":
        sizes = [n] * case["calls"] + ([case["last"]] if case["last"] else [])
        s.batches = [[img.copy() for img in _pictures(k, h, w, gen)] for k in sizes]
        return s
    # classifier inputs as the benchmark configurations state them: uniform where the network says so, else N(0, 1)
    uniform = case["net"] in ("vgg16", "alexnet_owt")
    make = torch.rand if uniform else torch.randn
    x = make((n, 3, h, w), generator=gen, device="cuda")
    if case["source"] == "array":
        s.x = x.cpu().numpy()
        return s
    s.x, p = _pinned(th, (n, 3, h, w))
    weakref.finalize(s, th.lib.THB200_HostFree, p)
    torch.from_numpy(s.x).copy_(x)
    s.result, s.ow, s.oh = C.POINTER(C.c_float)(), C.c_int(), C.c_int()
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------
def run(s):
    case, th = s.case, s.net.th
    if case["source"] == "images":
        outs = [th.process_images(s.net.handle, imgs)[0] for imgs in s.batches]
        return outs if len(outs) > 1 else outs[0]
    if case["source"] == "array":
        return th.process_float(s.net.handle, s.x)[0]
    n, c, h, w = s.x.shape
    count = th.lib.THProcessFloat(s.net.handle, s.x.ctypes.data, n, w, h, c, C.byref(s.result), C.byref(s.ow), C.byref(s.oh))
    if count <= 0:
        raise RuntimeError(th.lib.THB200_LastErrorString())
    return np.ctypeslib.as_array(s.result, shape=(count,))  # the network's own result buffer, as a C program reads it


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
# Output channels, kernel, stride and padding of every layer, to count with: (op, cout, k, stride, pad)
def _layers(net):
    if net == "alexnet_owt":
        return [("conv", 64, 11, 4, 2), ("pool", 0, 3, 2, 0), ("conv", 192, 5, 1, 2), ("pool", 0, 3, 2, 0), ("conv", 384, 3, 1, 1),
                ("conv", 256, 3, 1, 1), ("conv", 256, 3, 1, 1), ("pool", 0, 3, 2, 0), ("fc", 4096, 6, 1, 0), ("fc", 4096, 1, 1, 0),
                ("fc", 1000, 1, 1, 0)]
    out = []
    for ch, reps in ((64, 2), (128, 2), (256, 3), (512, 3), (512, 3)):
        out += [("conv", ch, 3, 1, 1)] * reps + [("pool", 0, 2, 2, 0)]
    return out + [("fc", 4096, 7, 1, 0), ("fc", 4096, 1, 1, 0), ("fc", 1000, 1, 1, 0)]


@functools.lru_cache(maxsize=256)
def _count(net, h, w, spatial):
    """(FLOPs of one image, weights, result values of one image)"""
    macs = weights = 0

    def conv(cin, cout, k, oh, ow):
        nonlocal macs, weights
        macs += cin * cout * k * k * oh * ow
        weights += cin * cout * k * k

    def out(v, k, s, p):
        return (v + 2 * p - k) // s + 1

    if net in ("resnet18", "resnet50"):
        h, w = out(h, 7, 2, 3), out(w, 7, 2, 3)
        conv(3, 64, 7, h, w)
        h, w, cin = out(h, 3, 2, 1), out(w, 3, 2, 1), 64
        for stage, reps in enumerate((2, 2, 2, 2) if net == "resnet18" else (3, 4, 6, 3)):
            mid = 64 << stage
            for r in range(reps):
                st = 2 if r == 0 and stage else 1
                oh, ow = out(h, 3, st, 1), out(w, 3, st, 1)
                if net == "resnet18":
                    conv(cin, mid, 3, oh, ow)
                    conv(mid, mid, 3, oh, ow)
                    cout = mid
                else:
                    conv(cin, mid, 1, h, w)
                    conv(mid, mid, 3, oh, ow)
                    cout = 4 * mid
                    conv(mid, cout, 1, oh, ow)
                if st != 1 or cin != cout:
                    conv(cin, cout, 1, oh, ow)
                h, w, cin = oh, ow, cout
        conv(cin, 1000, 1, 1, 1)
        return 2 * macs, weights, 1000
    if net == "segnet":
        cin, skips = 3, []
        for ch in (32, 64, 128, 256):
            conv(cin, ch, 3, h, w)
            skips.append(ch)
            h, w, cin = h // 2, w // 2, ch
        for i, ch in enumerate((128, 64, 32, 16)):
            conv(cin, ch, 4, h, w)  # transposed: every input pixel meets the whole kernel
            h, w, cin = 2 * h, 2 * w, ch + skips[3 - i]
        conv(cin, 21, 1, h, w)
        return 2 * macs, weights, 21 * h * w
    cin = 3
    for op, cout, k, st, p in _layers(net):
        h, w = out(h, k, st, p), out(w, k, st, p)
        if op != "pool":
            conv(cin, cout, k, h, w)
            cin = cout
    return 2 * macs, weights, cin * h * w


def _flops(net, h, w, spatial):
    return _count(net, h, w, spatial)[0]


def work(case):
    flops, weights, values = _count(case["net"], case["height"], case["width"], case["spatial"])
    images = case["batch"] * case["calls"] + case["last"]
    calls = case["calls"] + (1 if case["last"] else 0)
    per_image = 3 * case["height"] * case["width"] * (1 if case["source"] == "images" else 4)
    return {"bytes": images * (per_image + 4 * values) + calls * weights * WEIGHT_BYTES[case["mode"]], "flops": images * flops}


def tolerance(case):
    if case["mode"] == "int8":
        return "exact"
    # tens of layers, each rounding its output to the storage type once
    rel = {"fp32": 1e-5, "fp16": 4e-3, "bf16": 2e-2}[case["mode"]]
    if case["net"] == "alexnet_owt":
        rel = min(2.5 * rel, 2.5e-2)  # the soft-max turns the logits' absolute error into a relative one
    return {"rel": rel, "max": min(20 * rel, 0.5)}
