"""DK + DCN without kernel-space offsets outside the fp16 tensor-core kernels: the sampled kernel is laid out once per tap and channel.  Against the
oracle with offsets of zero: scopes that hit the cells and lie between them, runs of units that end inside a tap, one and two channels on a lane."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c,h,w,stride,k,scope,dtype", [
    (2, 40, 13, 17, 1, 3, (3, 3), torch.float32), (3, 24, 9, 10, 2, 3, (4, 4), torch.float32), (16, 96, 20, 20, 1, 3, (3, 3), torch.float32),
    (1, 8, 5, 3, 1, 3, (4, 3), torch.float32), (2, 72, 16, 12, 1, 3, (2, 3), torch.float32), (5, 104, 30, 31, 1, 3, (3, 3), torch.float16),
    (2, 40, 12, 15, 1, 2, (3, 4), torch.float32), (1, 33, 60, 70, 1, 3, (3, 3), torch.float32),
])
def test_shapes(n, c, h, w, stride, k, scope, dtype):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, k=k, scope=scope, stride=stride, pad=1, rot_std=0.5, off_std=2.0, seed=c + w)
    case["rotation"] = torch.zeros_like(case["rotation"])
    x, o, wt, dy = (case[i].to(dtype).cuda() for i in ("input", "offset", "weight", "grad_output"))
    leaves = [t.requires_grad_(True) for t in (x, o, wt)]
    y = deform_sample_depthwise(x, o, None, wt, **case["args"])
    got = (y.detach(),) + torch.autograd.grad(y, leaves, dy)
    a = [case[i].to(dtype).float() for i in ("grad_output", "input", "offset", "rotation", "weight")]
    back = O.deform_sample_depthwise_backward(*a, **case["args"])
    want = (O.deform_sample_depthwise_forward(*a[1:], **case["args"]), back[0], back[1], back[3])
    for name, g, v in zip(("output", "input", "offset", "weight"), got, want):
        assert rel_err(g, v.to(dtype)) < (1e-5 if dtype == torch.float32 else 2e-3), name


def test_values_that_are_not_finite():
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    case = make_case(2, 24, 12, 12, scope=(3, 3), rot_std=0.0, off_std=0.0, seed=3)
    x, o, wt, dy = (case[i].cuda() for i in ("input", "offset", "weight", "grad_output"))
    wt[7, 0, 1, 1] = float("inf")  # the cell of the middle tap; its neighbours read it with a weight of zero
    wt.requires_grad_(True)
    dy[1, 9, 4, 4] = float("nan")
    y = deform_sample_depthwise(x, o, None, wt, **case["args"])
    dw, = torch.autograd.grad(y, wt, dy)
    bad = ~torch.isfinite(y)
    assert bad[:, 7].any() and not bad[:, [c for c in range(24) if c != 7]].any()
    bad = ~torch.isfinite(dw)
    assert bad[9].any() and not bad[[c for c in range(24) if c != 9]].any()


@pytest.mark.parametrize("n,c,stride,dtype", [(2, 24, 1, torch.float32), (2, 64, 2, torch.float32), (3, 72, 1, torch.float16)])
def test_samples_outside_the_image_meet_no_value_that_is_not_finite(n, c, stride, dtype):
    """Finite wherever the oracle is: a tap that falls outside the image has no kernel value, whatever the bank holds."""
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, 12, 14, scope=(3, 3), stride=stride, rot_std=0.0, off_std=3.0, seed=c)
    case["weight"][7, 0, 0, 1], case["weight"][11, 0, 2, 2], case["weight"][c - 1, 0, 1, 0] = float("inf"), float("nan"), -float("inf")
    x, o, wt, dy = (case[i].to(dtype).cuda() for i in ("input", "offset", "weight", "grad_output"))
    leaves = [t.requires_grad_(True) for t in (x, o)]
    y = deform_sample_depthwise(x, o, None, wt, **case["args"])
    got = (y.detach(),) + torch.autograd.grad(y, leaves, dy)
    a = [case[i].to(dtype).float() for i in ("grad_output", "input", "offset", "rotation", "weight")]
    want = (O.deform_sample_depthwise_forward(*a[1:], **case["args"]),) + tuple(O.deform_sample_depthwise_backward(*a, **case["args"])[:2])
    for name, g, v in zip(("output", "input", "offset"), got, want):
        finite = torch.isfinite(v)
        assert (~finite).any() and finite.any(), name
        assert torch.isfinite(g.cpu()[finite]).all(), name
        assert rel_err(g.cpu()[finite], v[finite].to(dtype)) < (1e-5 if dtype == torch.float32 else 2e-3), name
