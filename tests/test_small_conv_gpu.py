"""Small fp16 calls of the local operator: block shapes of few channels and one item a warp, forward and grad-input, against the oracle.  Channels
with and without a remainder of 16, bands that end inside the plane, rows of odd width, planes smaller than an item, and sizes on both sides of
the line to the kernels for large calls."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,stride", [
    (1, 192, 28, 28, 1), (1, 160, 32, 32, 1), (1, 144, 56, 56, 2), (2, 64, 56, 56, 1), (1, 72, 24, 24, 1), (1, 104, 48, 48, 2), (1, 16, 9, 9, 1),
    (1, 40, 5, 200, 1), (3, 16, 1, 3, 1), (1, 8, 2, 2, 2), (1, 960, 7, 7, 1), (2, 312, 15, 18, 2), (3, 144, 56, 56, 1), (4, 144, 56, 56, 1), (1, 64, 96, 96, 2),
])
def test_small(n, c, h, w, stride):
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, stride=stride, pad=1, rot_std=0.7, seed=c + w)
    x, rot, wt, dy = (case[i].half().cuda() for i in ("input", "rotation", "weight", "grad_output"))
    x.requires_grad_(True)
    y = sample_depthwise(x, rot, wt, **case["args"])
    dx, = torch.autograd.grad(y, x, dy)
    a = [case[i].half().float() for i in ("grad_output", "input", "rotation", "weight")]
    want = (O.sample_depthwise_forward(*a[1:], **case["args"]), O.sample_depthwise_backward(*a, **case["args"])[0])
    for name, g, v in zip(("output", "input"), (y.detach(), dx), want):
        assert rel_err(g, v.half()) < 2e-3, name  # kernel values and results of 11 bits


@pytest.mark.parametrize("n,c,h,w,stride", [(2, 16, 28, 28, 1), (2, 32, 32, 32, 1), (2, 16, 56, 56, 2), (1, 32, 14, 17, 1), (2, 16, 9, 9, 2), (1, 64, 32, 64, 2), (2, 40, 24, 24, 1)])
def test_infinite_elements_on_the_border_stay_in_their_windows(n, c, h, w, stride):
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, stride=stride, pad=1, rot_std=0.7, seed=9)
    for t in (case["input"], case["grad_output"]):
        t[0, 3, 2, -1], t[0, 5, -1, 0], t[-1, 7, 0, 0] = float("inf"), float("-inf"), float("inf")
    x, rot, wt, dy = (case[i].half().cuda() for i in ("input", "rotation", "weight", "grad_output"))
    x.requires_grad_(True)
    y = sample_depthwise(x, rot, wt, **case["args"])
    dx, = torch.autograd.grad(y, x, dy)
    a = [case[i].half().float() for i in ("grad_output", "input", "rotation", "weight")]
    want = (O.sample_depthwise_forward(*a[1:], **case["args"]), O.sample_depthwise_backward(*a, **case["args"])[0])
    for name, g, v in zip(("output", "input"), (y.detach().float().cpu(), dx.float().cpu()), want):
        ok = torch.isfinite(v)
        assert 0 < int((~ok).sum()) <= 3 * 9 and torch.isfinite(g[ok]).all(), name
