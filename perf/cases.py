"""Timed cases of the mapped-operator path, called as a user's program calls it: `spherical_distortion.nn` modules (and
`spherical_distortion.functional` for the normalised scatter) on CUDA tensors, forward alone or forward and backward
through autograd.

Five kinds of work, every size in the case itself:

  layer       one MappedConvolution (3x3): an inner layer of a network, so the gradient of its input is wanted too
  stack       the four-layer spherical encoder: mapped convolutions with fused ReLU, strides 2, 2, 1, 1; its input is a
              batch of images, which take no gradient
  transposed  one MappedTransposedConvolution (3x3) doubling the resolution: a decoder layer
  pool        MappedMaxPool with indices, stride 2
  tangent     an equirectangular image gathered into 20 icosahedral tangent planes (Unresample) and, forward only,
              scattered back with weight-sum normalisation; or, in training, Unresample forward and backward

`precision` is what `_spherical_distortion_ext.set_precision` takes: "fp32" (the default) or "bf16" (tensor cores;
float32 tensors either way).  `map` is "gnomonic" (the kernel laid out on the sphere, what a spherical network uses) or
"random" (coordinates uniform over the image); `points` > 0 gives every kernel slot that many weighted points.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "spherical-package_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import _spherical_distortion_ext as ext  # noqa: E402
from spherical_distortion import functional as F  # noqa: E402
from spherical_distortion.nn import (InterpolationType, MappedConvolution, MappedMaxPool,  # noqa: E402
                                     MappedTransposedConvolution, Unresample)
from spherical_distortion.util import inverse_gnomonic_projection_map  # noqa: E402
from sphmap.workloads import tangent_image_map  # noqa: E402

KERNEL, K = 3, 9
STACK_STRIDES = (2, 2, 1, 1)
INTERP = {"nearest": InterpolationType.NEAREST, "bilinear": InterpolationType.BILINEAR,
          "bispherical": InterpolationType.BISPHERICAL}


# ---- cases ---------------------------------------------------------------------------------------------------------
def layer(name, precision, train, batch, cin, cout, height, width, map="gnomonic", interp="bilinear", points=0):
    return dict(name=name, kind="layer", precision=precision, train=train, batch=batch, cin=cin, cout=cout,
                height=height, width=width, map=map, interp=interp, points=points)


def stack(name, precision, train, batch, height, width, channels):
    return dict(name=name, kind="stack", precision=precision, train=train, batch=batch, height=height, width=width,
                channels=channels)


def transposed(name, precision, train, batch, cin, cout, height, width, map="gnomonic", interp="bilinear", points=0):
    return dict(name=name, kind="transposed", precision=precision, train=train, batch=batch, cin=cin, cout=cout,
                height=height, width=width, map=map, interp=interp, points=points)


def pool(name, train, batch, channels, height, width, map, interp):
    return dict(name=name, kind="pool", train=train, batch=batch, channels=channels, height=height, width=width,
                map=map, interp=interp)


def tangent(name, train, batch, channels, height, width, face):
    return dict(name=name, kind="tangent", train=train, batch=batch, channels=channels, height=height, width=width,
                face=face)


def listed():
    return [
        # the smallest call: one layer on a low-resolution panorama, forward only, default precision; launch latency
        layer("layer_forward_small", "fp32", False, 2, 16, 32, 64, 128),
        # a training step of a layer whose sizes fit no tile: odd channels, odd image, wrapped longitude
        layer("layer_train_ragged", "fp32", True, 3, 20, 37, 45, 91, interp="bispherical"),
        # an inner encoder layer trained in the default precision
        layer("layer_train_fp32", "fp32", True, 8, 64, 128, 128, 256),
        # weighted sampling: four points per kernel slot anywhere in the image, tensor-core precision
        layer("layer_train_weighted", "bf16", True, 16, 64, 128, 256, 512, map="random", interp="nearest", points=4),
        # one image through the encoder: inference latency
        stack("stack_infer_one", "bf16", False, 1, 512, 1024, 64),
        # a training step on one GPU's share of a batch that is split over eight
        stack("stack_train_shard", "bf16", True, 8, 512, 1024, 64),
        # the whole batch on one GPU: the largest step
        stack("stack_train", "bf16", True, 64, 512, 1024, 64),
        # a decoder layer trained in the default precision
        transposed("transposed_train_fp32", "fp32", True, 8, 128, 64, 128, 256),
        # pooling on a map without locality
        pool("pool_train_random", True, 8, 64, 256, 512, "random", "nearest"),
        # pooling between the layers of a spherical network, the module's default interpolation
        pool("pool_train_gnomonic", True, 16, 64, 256, 512, "gnomonic", "bilinear"),
        # a batch of RGB panoramas to tangent images and back
        tangent("tangent_roundtrip", False, 8, 3, 512, 1024, 64),
        # tangent images of high-resolution panoramas inside a network that is trained through them
        tangent("tangent_train_large", True, 32, 3, 1024, 2048, 256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, height):
    return 2 * height + rng.choice((0, 0, 0, 1, -3))


def _channels(rng, lo, hi):
    c = _log_int(rng, lo, hi)
    return c if rng.random() < 0.3 or c < 16 else c // 16 * 16  # mostly round counts, odd ones among them


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "stack", "stack", "transposed", "transposed", "pool", "pool", "tangent",
                       "tangent"))
    train = rng.random() < 0.6
    if kind == "tangent":
        h = _log_int(rng, 128, 1024)
        c = tangent("", train, _log_int(rng, 1, 32), rng.choice((1, 3, 3, 4, 7)), h, _width(rng, h), _log_int(rng, 16, 256))
    elif kind == "pool":
        h = _log_int(rng, 32, 320)
        c = pool("", train, _log_int(rng, 1, 16), _channels(rng, 3, 128), h, _width(rng, h),
                 rng.choice(("gnomonic", "gnomonic", "random")), rng.choice(("nearest", "bilinear")))
    elif kind == "stack":
        h = 4 * _log_int(rng, 16, 128)
        fp32 = rng.random() < 0.25
        c = stack("", "fp32" if fp32 else "bf16", train and not fp32, _log_int(rng, 1, 64), h, _width(rng, h),
                  rng.choice((32, 48, 64)))
        while work(c)["flops"] > (1.5e11 if fp32 else 1.2e13):
            c["batch"] = max(1, c["batch"] // 2)
            if c["batch"] == 1:
                c["height"], c["width"] = c["height"] // 2, c["width"] // 2
    else:
        h = _log_int(rng, 24, 256)
        weighted = rng.random() < 0.25
        c = (layer if kind == "layer" else transposed)(
            "", rng.choice(("fp32", "bf16")), train, _log_int(rng, 1, 16), _channels(rng, 3, 256), _channels(rng, 12, 256), h,
            _width(rng, h), "random" if weighted else "gnomonic", "nearest" if weighted else rng.choice(("bilinear", "bispherical")),
            4 if weighted else 0)
        # the exact precision runs at tens of TFLOP/s, the tensor cores at hundreds
        most = (5e10 if weighted else 1.5e11) if c["precision"] == "fp32" else 1.5e12
        while work(c)["flops"] > most:
            if c["batch"] > 1:
                c["batch"] //= 2
            else:
                c["cin"] = max(3, c["cin"] // 2)
    del c["name"]
    return c


# ---- geometry ------------------------------------------------------------------------------------------------------
def _half(n):
    return (n + 1) // 2


def _stack_layers(c):
    """(cin, cout, (IH, IW), (OH, OW), stride) of the four layers."""
    n = c["channels"]
    chans = (3, n, 2 * n, 4 * n, 4 * n)
    out, h, w = [], c["height"], c["width"]
    for i, s in enumerate(STACK_STRIDES):
        oh, ow = (_half(h), _half(w)) if s == 2 else (h, w)
        out.append((chans[i], chans[i + 1], (h, w), (oh, ow), s))
        h, w = oh, ow
    return out


def work(case):
    """Each input read once and each output written once; multiply-adds of the contractions count two."""
    c, f = case, 4
    if c["kind"] == "stack":
        ls = _stack_layers(c)
        fl = sum(2 * c["batch"] * co * ci * K * oh * ow for ci, co, _, (oh, ow), _ in ls)
        params = sum(co * ci * K + co for ci, co, _, _, _ in ls)
        maps = sum(oh * ow * K * 2 for _, _, _, (oh, ow), _ in ls)
        out = c["batch"] * ls[-1][1] * ls[-1][3][0] * ls[-1][3][1]
        nbytes = f * (c["batch"] * 3 * c["height"] * c["width"] + maps + params + out)
        if not c["train"]:
            return {"bytes": nbytes, "flops": fl}
        # the images take no gradient: two contractions of backward in every layer but the first, one there
        ci, co, _, (oh, ow), _ = ls[0]
        return {"bytes": nbytes + f * (out + params), "flops": 3 * fl - 2 * c["batch"] * co * ci * K * oh * ow}
    if c["kind"] in ("layer", "transposed"):
        big = c["height"] * c["width"]
        small = _half(c["height"]) * _half(c["width"])
        n_map, n_in, n_out = (big, big, big) if c["kind"] == "layer" else (small, small, big)
        pts = max(1, c["points"])
        fl = 2 * c["batch"] * c["cout"] * c["cin"] * K * n_map
        params = c["cin"] * c["cout"] * K + c["cout"]
        maps = n_map * K * pts * (3 if c["points"] else 2)
        x, y = c["batch"] * c["cin"] * n_in, c["batch"] * c["cout"] * n_out
        nbytes = f * (x + y + maps + params)
        return {"bytes": nbytes + f * (y + x + params), "flops": 3 * fl} if c["train"] else {"bytes": nbytes, "flops": fl}
    if c["kind"] == "pool":
        planes, n, o = c["batch"] * c["channels"], c["height"] * c["width"], _half(c["height"]) * _half(c["width"])
        nbytes = planes * (n * 4 + o * (4 + 8)) + o * K * 8
        return {"bytes": nbytes + (planes * (n * 4 + o * 4) if c["train"] else 0), "flops": planes * o * K}
    planes, n, o = c["batch"] * c["channels"], c["height"] * c["width"], 20 * c["face"] ** 2
    nbytes = planes * (min(4 * o, n) * 4 + o * 4) + o * 8 + planes * n * 4 + (planes * o * 4 if c["train"] else 0)
    return {"bytes": nbytes, "flops": planes * o * 14}


def tolerance(case):
    c = case
    if c["kind"] == "pool":
        return {"rel": 1e-6}  # values and indices are copies and comparisons; gradients sum a few float32 terms
    if c["kind"] == "tangent":
        return {"rel": 1e-6}  # a handful of float32 terms per value
    if c["precision"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3}  # float32 sums of up to a million terms
    # bf16 operands.  Through a trained stack a rounding can also switch a ReLU whose input is near zero.
    return {"rel": 2e-2 if c["kind"] == "stack" and c["train"] else 1e-2}


# ---- state ---------------------------------------------------------------------------------------------------------
def _map(c, gen, stride, points):
    """Sample map of the (height, width) image seen from its strided pixels, and interpolation weights or None."""
    h, w = c["height"], c["width"]
    if c["map"] == "gnomonic":
        return inverse_gnomonic_projection_map((h, w), (KERNEL, KERNEL), stride=stride, device="cuda"), None
    oh, ow = (_half(h), _half(w)) if stride == 2 else (h, w)
    size = torch.tensor([float(w), float(h)], device="cuda")
    if not points:
        return torch.rand(oh, ow, K, 2, generator=gen, device="cuda") * size, None
    m = torch.rand(oh, ow, K, points, 2, generator=gen, device="cuda") * size
    e = -torch.log(torch.rand(oh, ow, K, points, generator=gen, device="cuda").clamp_min(1e-12))
    return m, (e / e.sum(-1, keepdim=True)).contiguous()


def _init(module, fan, gen):
    with torch.no_grad():
        for p in (module.weight, module.bias):
            p.copy_((torch.rand(p.shape, generator=gen, device="cuda") * 2 - 1) / math.sqrt(fan))


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")  # noqa: E731
    uniform = lambda *shape: torch.rand(*shape, generator=gen, device="cuda")  # noqa: E731
    s = dict(c)
    b, h, w = c["batch"], c["height"], c["width"]
    if c["kind"] == "stack":
        s["modules"], s["maps"] = [], []
        for ci, co, hw, _, stride in _stack_layers(c):
            m = MappedConvolution(ci, co, K, InterpolationType.BILINEAR, activation="relu").cuda()
            _init(m, ci * K, gen)
            s["modules"].append(m)
            s["maps"].append(inverse_gnomonic_projection_map(hw, (KERNEL, KERNEL), stride=stride, device="cuda"))
        s["x"] = uniform(b, 3, h, w)
        if c["train"]:
            _, co, _, (oh, ow), _ = _stack_layers(c)[-1]
            s["grad"] = normal(b, co, oh, ow)
    elif c["kind"] == "layer":
        s["module"] = MappedConvolution(c["cin"], c["cout"], K, INTERP[c["interp"]]).cuda()
        _init(s["module"], c["cin"] * K, gen)
        s["map"], s["weights"] = _map(c, gen, 1, c["points"])
        s["x"] = normal(b, c["cin"], h, w).requires_grad_(c["train"])
        if c["train"]:
            s["grad"] = normal(b, c["cout"], h, w)
    elif c["kind"] == "transposed":
        s["module"] = MappedTransposedConvolution(c["cin"], c["cout"], K, INTERP[c["interp"]]).cuda()
        _init(s["module"], c["cin"] * K, gen)
        s["map"], s["weights"] = _map(c, gen, 2, c["points"])
        s["x"] = normal(b, c["cin"], _half(h), _half(w)).requires_grad_(c["train"])
        if c["train"]:
            s["grad"] = normal(b, c["cout"], h, w)
    elif c["kind"] == "pool":
        s["module"] = MappedMaxPool(K, INTERP[c["interp"]], return_indices=True)
        s["map"], _ = _map(c, gen, 2, 0)
        s["x"] = normal(b, c["channels"], h, w).requires_grad_(c["train"])
        if c["train"]:
            s["grad"] = normal(b, c["channels"], _half(h), _half(w))
    else:
        s["module"] = Unresample(InterpolationType.BILINEAR)
        s["map"] = tangent_image_map(h, w, c["face"]).cuda()
        s["x"] = uniform(b, c["channels"], h, w).requires_grad_(c["train"])
        if c["train"]:
            s["grad"] = normal(b, c["channels"], 20 * c["face"], c["face"])
    return s


# ---- one pass ------------------------------------------------------------------------------------------------------
def _backward(s, out, params):
    """One backward pass with fresh gradients, as after optimizer.zero_grad()."""
    for p in params:
        p.grad = None
    torch.autograd.backward([out], [s["grad"]])
    return [p.grad for p in params]


def run(state):
    s = state
    if s["kind"] == "pool":
        with torch.set_grad_enabled(s["train"]):
            out, idx = s["module"](s["x"], s["map"])
        return [out.detach(), idx] + (_backward(s, out, [s["x"]]) if s["train"] else [])
    if s["kind"] == "tangent":
        if s["train"]:
            out = s["module"](s["x"], s["map"])
            return [out.detach()] + _backward(s, out, [s["x"]])
        with torch.no_grad():
            faces = s["module"](s["x"], s["map"])
            back = F.resample_normalized(faces, s["map"], (s["height"], s["width"]), InterpolationType.BILINEAR)
        return [faces, back]
    ext.set_precision(s["precision"])
    with torch.set_grad_enabled(s["train"]):
        if s["kind"] == "stack":
            out, params = s["x"], []
            for m, sample_map in zip(s["modules"], s["maps"]):
                out = m(out, sample_map)
                params += [m.weight, m.bias]
        else:
            m = s["module"]
            params = [s["x"], m.weight, m.bias]
            if s["kind"] == "layer":
                out = m(s["x"], s["map"], s["weights"])
            else:
                out = m(s["x"], s["height"], s["width"], s["map"], s["weights"])
    return [out.detach()] + (_backward(s, out, params) if s["train"] else [])
