"""DK + DCN forward and gradients where the tensor-core kernels do not apply (fp32; fp16 with channels that are no multiple of
16, planes beyond 56 x 56, rows of odd width): remainders of the 32-channel groups, of the 32-pixel tiles and of the bands and pieces of rows,
single pixels, other strides, paddings and dilations, scopes other than 4 x 4, samples far outside, NaN offsets."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [
    (1, 1, 1, 1, 1, 1, 1, (4, 4)), (2, 33, 5, 40, 1, 1, 1, (4, 4)), (3, 8, 9, 7, 2, 1, 1, (3, 3)), (1, 72, 33, 35, 1, 2, 2, (2, 4)),
    (2, 24, 60, 61, 2, 0, 1, (4, 4)), (17, 40, 4, 4, 1, 1, 1, (1, 1)), (1, 8, 3, 120, 1, 1, 1, (6, 5)),
    (2, 96, 11, 13, 1, 1, 1, (4, 4)), (1, 128, 6, 8, 2, 1, 1, (4, 4)),
    (1, 40, 204, 210, 1, 1, 1, (4, 4)), (1, 34, 4, 700, 1, 1, 1, (3, 3))]  # no room for the sort or the sums of grad-input


@pytest.mark.parametrize("n,c,h,w,stride,pad,dil,scope", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_gradients(n, c, h, w, stride, pad, dil, scope, dtype):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, scope=scope, stride=stride, pad=pad, dil=dil, rot_std=0.8, off_std=1.5, seed=c + h)
    if h > 4:
        case["offset"][0, 0, 0, 0], case["offset"][0, 3, -1, -1], case["offset"][0, 8, 1, 1] = float("nan"), 1e9, -float("inf")
    x, o, r, wt, dy = (case[k].to(dtype).to(DEV) for k in ("input", "offset", "rotation", "weight", "grad_output"))
    leaves = [t.requires_grad_(True) for t in (x, o, r, wt)]
    y = deform_sample_depthwise(*leaves, **case["args"])
    got = torch.autograd.grad(y, leaves, dy)
    # beyond 128 pixels fp32 rounds a coordinate at 2^-17 and more: samples (and cells, at the floor) are those of the fp32 oracle
    up = torch.float32 if dtype == torch.float16 or max(h, w) > 128 else torch.float64
    a = [case[k].to(dtype).to(up) for k in ("grad_output", "input", "offset", "rotation", "weight")]
    want = O.deform_sample_depthwise_backward(*a, **case["args"])
    tol = 2e-3 if dtype == torch.float16 else 1e-5
    want = (O.deform_sample_depthwise_forward(*a[1:], **case["args"]), *want)
    for g, w in zip((y.detach(), *got), want):
        assert rel_err(g, w.to(dtype)) < tol


@pytest.mark.parametrize("h,w", [(90, 91), (105, 112), (127, 95)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_planes_whose_cells_take_32_to_48_kilobytes(h, w, dtype):
    """The sort's counters and its static arrays together take more shared memory than a launch has without asking."""
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(1, 24, h, w, scope=(4, 4), rot_std=0.5, off_std=2.0, seed=h)
    names = ("grad_output", "input", "offset", "rotation", "weight")
    want = O.deform_sample_depthwise_backward(*(case[k].to(dtype).float() for k in names), **case["args"])
    dy, *leaves = (case[k].to(dtype).to(DEV) for k in names)
    leaves = [t.requires_grad_(True) for t in leaves]
    got = torch.autograd.grad(deform_sample_depthwise(*leaves, **case["args"]), leaves, dy)
    for g, v in zip(got, want):
        assert rel_err(g, v.to(dtype)) < (1e-5 if dtype == torch.float32 else 2e-3)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_subsets_of_the_gradients_agree(dtype):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    case = make_case(2, 72, 11, 13, rot_std=0.8, off_std=1.5, seed=5)
    x, o, r, wt, dy = (case[k].to(dtype).to(DEV) for k in ("input", "offset", "rotation", "weight", "grad_output"))
    leaves = [t.requires_grad_(True) for t in (x, o, r, wt)]
    full = torch.autograd.grad(deform_sample_depthwise(*leaves, **case["args"]), leaves, dy)
    for i, leaf in enumerate(leaves):
        args = [t if t is leaf else t.detach() for t in leaves]
        one, = torch.autograd.grad(deform_sample_depthwise(*args, **case["args"]), [leaf], dy)
        assert rel_err(one, full[i]) < (2e-3 if dtype == torch.float16 else 1e-5)


@pytest.mark.parametrize("c,scope", [(40, (3, 3)), (24, (6, 5)), (128, (3, 3))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_without_kernel_offsets(c, scope, dtype):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    case = make_case(2, c, 12, 9, scope=scope, off_std=1.5, seed=7)
    x, o, r, wt, dy = (case[k].to(dtype).to(DEV) for k in ("input", "offset", "rotation", "weight", "grad_output"))
    leaves = [t.requires_grad_(True) for t in (x, o, wt)]
    a = deform_sample_depthwise(x, o, torch.zeros_like(r), wt, **case["args"])
    b = deform_sample_depthwise(x, o, None, wt, **case["args"])
    for p, q in zip((a, *torch.autograd.grad(a, leaves, dy)), (b, *torch.autograd.grad(b, leaves, dy))):
        assert rel_err(q, p) < (2e-3 if dtype == torch.float16 else 1e-5)


@pytest.mark.parametrize("c", [40, 24, 104])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_values_that_are_not_finite_stay_where_they_belong(c, dtype):
    """Wherever the oracle is finite, all gradients together and the bank gradient alone are finite and agree (offsets that leave the
    first row and column of taps of an image outside it, and let each tap touch four known cells of the bank)."""
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(2, c, 12, 9, rot_std=0.05, off_std=0.05, seed=22)
    case["rotation"] += 0.25
    case["offset"] -= 0.3
    case["weight"][5, 0, 0, 0] = float("inf")
    case["grad_output"][0, 3, 0, 0], case["input"][1, 9, 0, 0] = float("inf"), -float("inf")
    a = [case[k].to(dtype) for k in ("grad_output", "input", "offset", "rotation", "weight")]
    dy, *leaves = (t.to(DEV) for t in a)
    for t in leaves:
        t.requires_grad_(True)
    y = deform_sample_depthwise(*leaves, **case["args"])
    got = (y.detach(),) + torch.autograd.grad(y, leaves, dy)
    d = [t.double() for t in a]
    want = (O.deform_sample_depthwise_forward(*d[1:], **case["args"]), *O.deform_sample_depthwise_backward(*d, **case["args"]))
    alone, = torch.autograd.grad(deform_sample_depthwise(*[t.detach() for t in leaves[:3]], leaves[3], **case["args"]), [leaves[3]], dy)
    for g, v in zip((*got, alone), (*want, want[-1])):
        ok = torch.isfinite(v)
        assert 0 < int((~ok).sum()) and int(ok.sum()) > v.numel() // 4
        g = g.double().cpu()
        assert torch.isfinite(g[ok]).all()
        assert float((g[ok] - v[ok]).norm() / v[ok].norm()) < (2e-3 if dtype == torch.float16 else 1e-5)
