"""DK + DCN bank and input gradients where the tensor-core kernels do not apply (fp32; fp16 with channels that are no multiple of
16 or planes beyond 56 x 56): remainders of the 32-channel groups, of the 32-pixel tiles and of the bands and pieces of rows,
single pixels, other strides, paddings and dilations, scopes other than 4 x 4, samples far outside, NaN offsets."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [
    (1, 1, 1, 1, 1, 1, 1, (4, 4)), (2, 33, 5, 40, 1, 1, 1, (4, 4)), (3, 8, 9, 7, 2, 1, 1, (3, 3)), (1, 72, 33, 35, 1, 2, 2, (2, 4)),
    (2, 24, 60, 61, 2, 0, 1, (4, 4)), (17, 40, 4, 4, 1, 1, 1, (1, 1)), (1, 8, 3, 120, 1, 1, 1, (6, 5))]


@pytest.mark.parametrize("n,c,h,w,stride,pad,dil,scope", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_input_and_bank_gradient(n, c, h, w, stride, pad, dil, scope, dtype):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, scope=scope, stride=stride, pad=pad, dil=dil, rot_std=0.8, off_std=1.5, seed=c + h)
    if h > 4:
        case["offset"][0, 0, 0, 0], case["offset"][0, 3, -1, -1], case["offset"][0, 8, 1, 1] = float("nan"), 1e9, -float("inf")
    x, o, r, wt, dy = (case[k].to(dtype).to(DEV) for k in ("input", "offset", "rotation", "weight", "grad_output"))
    x.requires_grad_(True), wt.requires_grad_(True)
    dx, dw = torch.autograd.grad(deform_sample_depthwise(x, o, r, wt, **case["args"]), [x, wt], dy)
    up = torch.float32 if dtype == torch.float16 else torch.float64
    a = [case[k].to(dtype).to(up) for k in ("grad_output", "input", "offset", "rotation", "weight")]
    want = O.deform_sample_depthwise_backward(*a, **case["args"])
    tol = 2e-3 if dtype == torch.float16 else 1e-5
    assert rel_err(dx, want[0].to(dtype)) < tol
    assert rel_err(dw, want[3].to(dtype)) < tol
