"""The local operator with any number of channels, against the CPU oracle: fp32 runs on the tcgen05 kernels (one channel per
TMEM lane), fp16 there on wide rows, else on the mma.sync kernels (channels a multiple of 16) or the general ones.  The sizes are the
edges of their tiles: 32-channel groups (1 to 5 of them, full and partial, so that every placement of the remaining groups on the
lanes occurs), 8-pixel segments, rows with and without TMA, planes of one row or one pixel, steps that span samples, more channels
than one block takes."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [
    (1, 8, 1, 1), (5, 16, 1, 9), (3, 24, 7, 7), (2, 32, 8, 8), (2, 40, 9, 16), (1, 56, 17, 24), (2, 72, 19, 23),
    (1, 104, 12, 33), (2, 136, 5, 40), (1, 160, 28, 28), (1, 200, 14, 14), (1, 264, 3, 64), (9, 280, 4, 4), (1, 1096, 6, 10),
    (1, 24, 112, 112), (1, 8, 2, 200), (1, 32, 110, 110), (2, 48, 31, 57),
    (2, 72, 31, 48), (5, 264, 2, 32), (2, 72, 9, 28), (1, 40, 5, 36), (2, 104, 6, 100),
    (1, 16, 9, 73), (1, 32, 7, 97), (2, 48, 5, 101), (1, 96, 6, 111),  # rows of odd width, a warp per row and not
    (13, 24, 57, 58), (13, 8, 113, 114),  # few channels, the GPU full
]


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("n,c,h,w", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_shapes(n, c, h, w, stride, dtype):
    _check(make_case(n, c, h, w, stride=stride, rot_std=1.0, seed=c + w), dtype)


@pytest.mark.parametrize("scope", [(1, 1), (2, 2), (3, 3), (3, 5), (2, 8)])
def test_scopes(scope):
    _check(make_case(2, 40, 11, 18, scope=scope, rot_std=1.0, seed=3), torch.float32)


@pytest.mark.parametrize("scale", [1e-30, 1e-6, 1e6, 1e30])
def test_bank_magnitudes(scale):
    """fp32 banks are split into scaled fp16 pieces, each channel by its own power of two."""
    case = make_case(2, 48, 9, 17, rot_std=1.0, seed=5)
    case["weight"] *= scale ** torch.linspace(-0.5, 1, 48).view(48, 1, 1, 1)
    x, r, w = (case[k].to(DEV) for k in ("input", "rotation", "weight"))
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    y = sample_depthwise(x, r, w, **case["args"])
    want = O.sample_depthwise_forward(*(case[k].double() for k in ("input", "rotation", "weight")), **case["args"])
    per = (y.double().cpu() - want).abs().amax((0, 2, 3)) / want.abs().amax((0, 2, 3))
    assert float(per.max()) < 1e-5


@pytest.mark.parametrize("n,c,h,w,stride", [(2, 64, 28, 28, 1), (2, 144, 30, 37, 2), (3, 960, 7, 7, 1)])
def test_error_against_fp64(n, c, h, w, stride):
    """2-norm error of fp32 results.  Forward and grad-input: a coordinate between 1 and 4 is rounded at 2^-24 to 2^-22, which moves a
    kernel value by 1.3e-7 of its size, the sampled kernel itself is off by 4.5e-8, products and store by 4e-8: 1.4e-7 in all for four
    gathered fp32 products as for the split ones, here with a tenth more.  Offsets: chains of C / 8 + 39 additions at
    8.6e-8 sqrt(L / 24), beside 8e-8; a tenth more."""
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, stride=stride, rot_std=1.0, seed=c)
    x, r, wt, dy = (case[k].to(DEV) for k in ("input", "rotation", "weight", "grad_output"))
    for t in (x, r):
        t.requires_grad_(True)
    y = sample_depthwise(x, r, wt, **case["args"])
    got = (y.detach(),) + torch.autograd.grad(y, [x, r], dy)
    a = {k: case[k].double() for k in ("input", "rotation", "weight", "grad_output")}
    want = (O.sample_depthwise_forward(a["input"], a["rotation"], a["weight"], **case["args"]),)
    want += tuple(O.sample_depthwise_backward(a["grad_output"], a["input"], a["rotation"], a["weight"], **case["args"])[:2])
    chain = 1.1 * ((8e-8) ** 2 + (8.6e-8) ** 2 * (c / 8 + 39) / 24) ** 0.5
    for name, g, v, bound in zip(("output", "grad_input", "grad_rotation"), got, want, (1.55e-7, 1.55e-7, chain)):
        err = float((g.double().cpu() - v).norm() / v.norm())
        assert err < bound, "%s %.3e (bound %.3e)" % (name, err, bound)


@pytest.mark.parametrize("stride", [1, 2])
def test_wide_range_inside_a_channel(stride):
    """Cells from 1 down to 2^-40 of the channel's largest, sampled with offsets that are multiples of 1/64 (hat products exact).  The
    sums of products are truncated five times at 2^-23 and the nine products with the input add ten roundings: 2^-20 of the sum of
    magnitudes.  The pieces of the bank end at 2^-54 of the largest cell, and products with a hat of zero still take part in the
    alignment of a sum (2^-53 of it seen): 2^-50 of the largest cell."""
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(2, 40, 13, 21, stride=stride, rot_std=1.0, seed=8)
    gen = torch.Generator().manual_seed(9)
    w = case["weight"] * torch.exp2(-40 * torch.rand(case["weight"].shape, generator=gen))
    r = torch.round(case["rotation"] * 64) / 64
    r[0] = torch.round(r[0])  # one cell alone
    x, dy = case["input"], case["grad_output"]
    xg = x.to(DEV).requires_grad_(True)
    y = sample_depthwise(xg, r.to(DEV), w.to(DEV), **case["args"])
    dx, = torch.autograd.grad(y, [xg], dy.to(DEV))

    def both(x, r, w, dy):
        args = [t.double() for t in (dy, x, r, w)]
        return O.sample_depthwise_forward(*args[1:], **case["args"]), O.sample_depthwise_backward(*args, **case["args"])[0]
    flat = w.abs().amax((2, 3), keepdim=True).expand_as(w)
    for got, want, size, top in zip((y.detach(), dx), both(x, r, w, dy), both(x.abs(), r, w.abs(), dy.abs()),
                                    both(x.abs(), torch.zeros_like(r), flat, dy.abs())):
        over = (got.double().cpu() - want).abs() - (2.0 ** -20 * size + 2.0 ** -50 * top)
        assert float(over.max()) <= 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("c,h,w,stride", [(40, 9, 24, 1), (40, 10, 24, 2), (136, 7, 28, 1), (24, 9, 13, 2)])
def test_values_that_are_not_finite_stay_where_they_belong(c, h, w, stride, dtype):
    """Wherever the oracle is finite, results are finite and agree: a bank cell reaches the outputs and gradients of the samples that
    touch it, an input or upstream gradient the cells that its samples touch (kernel offsets near 1/4, so that each tap touches four
    known cells, and the taps in the padding none)."""
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(2, c, h, w, stride=stride, rot_std=0.05, seed=21)
    case["rotation"] += 0.25
    case["weight"][5, 0, 0, 0], case["weight"][c - 1, 0, 2, 1] = float("inf"), float("nan")
    case["grad_output"][0, 3, 0, 0], case["input"][1, 9, 0, 0] = float("inf"), -float("inf")
    a = {k: case[k].to(dtype) for k in ("input", "rotation", "weight", "grad_output")}
    x, r, wt, dy = (a[k].to(DEV) for k in ("input", "rotation", "weight", "grad_output"))
    for t in (x, r, wt):
        t.requires_grad_(True)
    y = sample_depthwise(x, r, wt, **case["args"])
    got = (y.detach(),) + torch.autograd.grad(y, [x, r, wt], dy)
    d = {k: v.double() for k, v in a.items()}
    want = [O.sample_depthwise_forward(d["input"], d["rotation"], d["weight"], **case["args"])]
    want += O.sample_depthwise_backward(d["grad_output"], d["input"], d["rotation"], d["weight"], **case["args"])
    for g, v in zip(got, want):
        ok = torch.isfinite(v)
        assert 0 < int((~ok).sum()) and int(ok.sum()) > v.numel() // 4
        g = g.double().cpu()
        assert torch.isfinite(g[ok]).all()
        assert float((g[ok] - v[ok]).norm() / v[ok].norm()) < (2e-3 if dtype == torch.float16 else 1e-5)


def _flat(t, skip):
    """A copy of t that starts `skip` elements into its storage."""
    out = torch.empty(t.numel() + skip, dtype=t.dtype, device=t.device)[skip:].view(t.shape)
    return out.copy_(t)


@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("n,c,h,w,stride", [(2, 24, 20, 24, 1), (2, 40, 11, 64, 2), (1, 72, 9, 28, 1), (2, 72, 13, 101, 1), (3, 104, 7, 7, 2)])
def test_fp16_channels_no_multiple_of_16_are_computed_in_fp32(n, c, h, w, stride, skip):
    """Results are off by their rounding to fp16 only: relative 2^-12 / sqrt(3) to 2^-11 / sqrt(3) depending on the mantissa, 2.1e-4 over
    a binade, here with a fifth more (kernel values or products rounded to fp16: 3e-4 to 3.6e-4).  Products dy x beyond 65504 are no
    limit either.  skip = 1: tensors on odd addresses."""
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, stride=stride, rot_std=1.0, seed=c)
    half = {k: case[k].half() for k in ("input", "rotation", "weight", "grad_output")}

    def run(a):
        x, r, wt, dy = (_flat(a[k].to(DEV), skip) for k in ("input", "rotation", "weight", "grad_output"))
        for t in (x, r, wt):
            t.requires_grad_(True)
        y = sample_depthwise(x, r, wt, **case["args"])
        d = {k: v.double() for k, v in a.items()}
        want = [O.sample_depthwise_forward(d["input"], d["rotation"], d["weight"], **case["args"])]
        want += O.sample_depthwise_backward(d["grad_output"], d["input"], d["rotation"], d["weight"], **case["args"])
        return zip(("output", "grad_input", "grad_rotation", "grad_weight"), (y.detach(),) + torch.autograd.grad(y, [x, r, wt], dy), want)
    for name, g, v in run(half):
        err = float((g.double().cpu() - v).norm() / v.norm())
        assert err < 2.5e-4, "%s %.2e" % (name, err)
    half["input"] = half["input"] * 128
    half["grad_output"] = half["grad_output"] * 128
    half["weight"] = half["weight"] / 128
    assert float(half["input"].abs().max()) * float(half["grad_output"].abs().max()) > 65504
    for name, g, v in run(half):
        if name == "grad_rotation":
            assert float((g.double().cpu() - v).norm() / v.norm()) < 2.5e-4


def test_offsets_that_sample_nothing():
    case = make_case(1, 40, 9, 20, rot_std=1.0, seed=6)
    r = case["rotation"]
    r[0, 0, 2] = float("nan")
    r[0, 5, 3] = float("inf")
    r[0, 9, 4] = 1e30
    r[0, 12] = -7.0
    x, rr, w = (case[k].to(DEV) for k in ("input", "rotation", "weight"))
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    y = sample_depthwise(x, rr, w, **case["args"])
    case["rotation"] = torch.nan_to_num(r, nan=50.0, posinf=50.0)
    want = O.sample_depthwise_forward(*(case[k].double() for k in ("input", "rotation", "weight")), **case["args"])
    assert rel_err(y, want) < 1e-5


def test_every_kernel_has_the_registers_of_its_roles():
    """setmaxnreg moves registers between warps; what the shares add up to has to be there in every instantiation."""
    import ctypes
    from deformable_kernels import _cabi as C
    out = (ctypes.c_longlong * 8)()
    g = C.geom((1, 16, 8, 8), (3, 3), (1, 1), (1, 1), (1, 1), (4, 4), 1)
    assert C.lib.dk_local_plan_query(g, C.DK_F32, 8, out) == 0
    assert out[0] >= 32 and out[1] >= out[2] >= 72


def _check(case, dtype):
    from deformable_kernels import _cabi as C
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    x, r, w, dy = (case[k].to(dtype).to(DEV) for k in ("input", "rotation", "weight", "grad_output"))
    for t in (x, r, w):
        t.requires_grad_(True)
    y = sample_depthwise(x, r, w, **case["args"])
    got = [y.detach()] + list(torch.autograd.grad(y, [x, r, w], dy))
    up = torch.float32 if dtype == torch.float16 else torch.float64
    a = {k: case[k].to(dtype).to(up) for k in ("input", "rotation", "weight", "grad_output")}
    want = [O.sample_depthwise_forward(a["input"], a["rotation"], a["weight"], **case["args"])]
    want += list(O.sample_depthwise_backward(a["grad_output"], a["input"], a["rotation"], a["weight"], **case["args"]))
    tol = 2e-3 if dtype == torch.float16 else 1e-5
    for name, g, v in zip(("output", "grad_input", "grad_rotation", "grad_weight"), got, want):
        assert rel_err(g, v.to(dtype)) < tol, "%s %.2e" % (name, rel_err(g, v.to(dtype)))
    assert C.lib.dk_ring_error_status() == 0
