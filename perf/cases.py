"""The work that users of the deformable-kernel operators have them do, as cases that can be timed.

A case goes through the public entry points (`sample_depthwise`, `deform_sample_depthwise`, `nd_linear_sample` and the
`GlobalDeformKernel2d` layer) the way a training loop (forward, then every gradient) or an inference service (forward
under `no_grad`) calls them.  Tensors hold what such programs put there: N(0, 1) activations and upstream gradients,
kaiming-scaled weight banks, kernel-space offsets of 0.5 to 1 cell, image-space offsets of 2 pixels.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("deformable-kernels_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from deformable_kernels.modules import GlobalDeformKernel2d  # noqa: E402
from deformable_kernels.ops.deform_kernel.functions import (  # noqa: E402
    deform_sample_depthwise, nd_linear_sample, sample_depthwise)

_DTYPES = {"fp16": torch.float16, "fp32": torch.float32}


def _local(name, n, c, h, w, stride, dtype, grad=True, scope=4):
    return dict(name=name, op="local", n=n, c=c, h=h, w=w, stride=stride, scope=scope, dtype=dtype, grad=grad)


def _deform(name, n, c, h, w, stride, dtype, rotation, scope, grad=True):
    return dict(name=name, op="deform", n=n, c=c, h=h, w=w, stride=stride, scope=scope, dtype=dtype, grad=grad,
                rotation=rotation)


def _global(name, n, c, h, w, scope, dtype, grad=True):
    return dict(name=name, op="global", n=n, c=c, h=h, w=w, scope=scope, dtype=dtype, grad=grad)


def _nd(name, c, b, dims, scope, dtype, grad=True):
    return dict(name=name, op="nd", c=c, b=b, dims=dims, scope=scope, dtype=dtype, grad=grad)


def listed():
    return [
        # one image through one layer of a service: nothing but latency
        _local("local_fp16_one_image", 1, 192, 28, 28, 1, "fp16", grad=False),
        # the small fp32 layer that a first experiment or a gradient check starts from
        _local("local_fp32_small", 2, 64, 28, 28, 1, "fp32"),
        # the layer sweep of a mobile classification network at 224 x 224, batch 128, mixed precision: its largest layer,
        # a downsampling layer, and two of the many layers on small planes
        _local("local_fp16_c96_112", 128, 96, 112, 112, 1, "fp16"),
        _local("local_fp16_c144_56_s2", 128, 144, 56, 56, 2, "fp16"),
        _local("local_fp16_c384_14", 128, 384, 14, 14, 1, "fp16"),
        _local("local_fp16_c960_7_s2", 128, 960, 7, 7, 2, "fp16"),
        # dense prediction on images that are no multiple of anything, few images per GPU, channels a multiple of 8
        _local("local_fp16_ragged", 8, 72, 75, 101, 1, "fp16"),
        # full precision, as the operators run under mixed precision tools that keep them in fp32
        _local("local_fp32_c144_56", 64, 144, 56, 56, 1, "fp32"),
        # kernel-space and image-space offsets together
        _deform("deform_fp16_c256_56", 64, 256, 56, 56, 1, "fp16", True, 4),
        # a depthwise deformable convolution (no kernel-space offsets, scope = kernel) in full precision
        _deform("deform_fp32_c192_28", 16, 192, 28, 28, 1, "fp32", False, 3),
        # one resampled kernel per sample: the layer, and the N-d sampler as a 3 x 3 kernel's layer calls it
        _global("global_fp32_c256_14", 32, 256, 14, 14, 2, "fp32"),
        _nd("nd_fp32_c256", 256, 288, 2, 4, "fp32"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Batches of 1 to 128, planes of 7 to 112 rows of a similar number of columns, channels in multiples of 8 from 16 to
    960 (the rounding that width-scaled networks use), both strides, both precisions, training and inference."""
    op = rng.choice(["local"] * 6 + ["deform"] * 2 + ["global", "nd"])
    dtype = rng.choice(["fp16", "fp16", "fp32"])
    grad = rng.random() < 0.75
    if op == "nd":
        dims = rng.choice([1, 2, 2, 2, 3])
        c = _log_int(rng, 16, 4096)
        case = _nd("", c, min(_log_int(rng, 1, 4096), (1 << 22) // c), dims, rng.randint(2, 5), "fp32", grad)
    else:
        c = 8 * _log_int(rng, 2, 120)
        h = _log_int(rng, 7, 112)
        w = max(7, min(112, int(round(h * rng.uniform(0.6, 1.6)))))
        most = (1 << 23) if op == "deform" or dtype == "fp32" else (3 << 23)  # input elements
        n = max(1, min(_log_int(rng, 1, 128), most // (c * h * w)))
        stride = rng.choice([1, 1, 2])
        if op == "local":
            case = _local("", n, c, h, w, stride, dtype, grad)
        elif op == "deform":
            rotation = rng.random() < 0.5
            case = _deform("", n, c, h, w, stride, dtype, rotation, 4 if rotation else 3, grad)
        else:
            case = _global("", n, c, h, w, rng.choice([2, 3, 4]), dtype, grad)
    del case["name"]
    return case


def _out(i, stride):
    return (i - 1) // stride + 1  # kernel 3, padding 1


class _Draw:
    def __init__(self, seed, dtype, grad):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.dtype, self.grad = dtype, grad

    def normal(self, *shape, std=1.0, leaf=True):
        t = torch.randn(*shape, device="cuda", dtype=self.dtype, generator=self.gen)
        if std != 1.0:
            t.mul_(std)
        return t.requires_grad_(self.grad and leaf)

    def uniform(self, lo, hi, *shape):
        t = torch.rand(*shape, device="cuda", dtype=self.dtype, generator=self.gen)
        return t.mul_(hi - lo).add_(lo).requires_grad_(self.grad)


def prepare(case, seed):
    op, grad, s = case["op"], case["grad"], case["scope"]
    d = _Draw(seed, _DTYPES[case["dtype"]], grad)
    state = dict(case=case)
    if op == "nd":
        c, b, dims = case["c"], case["b"], case["dims"]
        state["inputs"] = [d.normal(c, *[s] * dims, std=math.sqrt(2.0 / s ** dims)), d.uniform(0.0, s - 1.0, b, dims)]
        state["dy"] = d.normal(b, c, leaf=False)
        return state
    n, c, h, w = case["n"], case["c"], case["h"], case["w"]
    x = d.normal(n, c, h, w)
    if op == "global":
        layer = GlobalDeformKernel2d((s, s), c, c, kernel_size=1, groups=c).cuda()
        params = _Draw(seed + 1, torch.float32, False)
        with torch.no_grad():
            layer.weight.copy_(params.normal(*layer.weight.shape, std=math.sqrt(2.0 / (s * s))))
            layer.fc.weight.copy_(params.normal(*layer.fc.weight.shape, std=0.5))
            layer.fc.bias.copy_(params.normal(*layer.fc.bias.shape, std=0.1))
        layer.requires_grad_(grad)
        state["layer"], state["inputs"] = layer, [x, layer.weight, layer.fc.weight, layer.fc.bias]
        state["dy"] = d.normal(n, c, h, w, leaf=False)
        return state
    st = case["stride"]
    ho, wo = _out(h, st), _out(w, st)
    bank = d.normal(c, 1, s, s, std=math.sqrt(2.0 / (s * s)))
    if op == "local":
        state["inputs"] = [x, d.normal(n, 18, ho, wo), bank]
    else:
        rotation = d.normal(n, 18, ho, wo, std=0.5) if case["rotation"] else None
        state["inputs"] = [x, d.normal(n, 18, ho, wo, std=2.0), rotation, bank]
    state["dy"] = d.normal(n, c, ho, wo, leaf=False)
    return state


def _forward(state):
    case, inputs = state["case"], state["inputs"]
    if case["op"] == "local":
        return sample_depthwise(*inputs, (3, 3), (case["stride"],) * 2, (1, 1))
    if case["op"] == "deform":
        return deform_sample_depthwise(*inputs, (3, 3), (case["stride"],) * 2, (1, 1))
    if case["op"] == "global":
        return state["layer"](inputs[0])
    return nd_linear_sample(*inputs)


def run(state):
    if not state["case"]["grad"]:
        with torch.no_grad():
            return _forward(state)
    y = _forward(state)
    return (y,) + torch.autograd.grad(y, [t for t in state["inputs"] if t is not None], state["dy"])


def work(case):
    """Every input read once and every output written once per direction, the saved inputs read again by the backward."""
    e = 2 if case["dtype"] == "fp16" else 4
    op, grad, s = case["op"], case["grad"], case["scope"]
    if op == "nd":
        cells, out = case["c"] * s ** case["dims"], case["b"] * case["c"]
        coord, corners = case["b"] * case["dims"], 2 ** case["dims"]
        nbytes = cells + coord + out + (2 * (cells + coord) + out if grad else 0)
        return {"bytes": nbytes * 4, "flops": out * 2 * corners * ((2 + case["dims"]) if grad else 1)}
    n, c, h, w = case["n"], case["c"], case["h"], case["w"]
    x, bank = n * c * h * w, c * s * s
    if op == "global":
        params = (bank + 2 * c + 4) * 4
        nbytes = 2 * x * e + params + ((3 * x * e + 2 * params) if grad else 0)
        return {"bytes": nbytes, "flops": x * (5 if grad else 2)}
    ho, wo = _out(h, case["stride"]), _out(w, case["stride"])
    y, planes = n * c * ho * wo, 18 * n * ho * wo
    kernel_offsets = op == "local" or case["rotation"]
    offsets = planes * (int(kernel_offsets) + int(op == "deform"))
    nbytes = x + y + offsets + bank + ((2 * x + y + 2 * (offsets + bank)) if grad else 0)
    # per output and tap: the resampled kernel value (4 multiply-adds; once for all pixels where it is the bank itself),
    # the sampled image value (4), their product; backward the same values once more and the gradients towards the image,
    # the bank and the offsets
    k, i = 4 * int(kernel_offsets), 4 * int(op == "deform")
    fma = k + i + 1
    if grad:
        fma += k + i + (1 + max(1, i)) + (1 + max(1, k)) + k + i
    return {"bytes": nbytes * e, "flops": 2 * 9 * y * fma}


def tolerance(case):
    """fp16: results rounded to fp16 (2^-11), as may be the resampled kernel and the products that feed a matrix
    instruction.  fp32: sums of up to some 10^5 terms in another order.  Largest differences: single elements whose terms
    cancel, against the tensor's own scale."""
    if case["dtype"] == "fp16":
        return {"rel": 2e-3, "max": 5e-2}
    return {"rel": 1e-5, "max": 5e-4}
