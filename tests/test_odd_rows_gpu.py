"""fp16 band kernels, mostly at stride 2 on rows of odd width from 71 to 97 columns, on either side of the line from which rows are copied word by word:
planes that start on an even or odd half, bands at both ends of a plane, blocks of one and of several slabs of channels."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu


def _odd_start(t):
    """The same values one half behind an aligned address."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return buf[1:].view(t.shape).copy_(t)


def _check(n, c, h, w, stride, shifted):
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    from oracle import dk_oracle as O
    case = make_case(n, c, h, w, stride=stride, rot_std=0.7, seed=c + w)
    x, r, k, dy = (case[name].half() for name in ("input", "rotation", "weight", "grad_output"))
    want = (O.sample_depthwise_forward(x.float(), r.float(), k.float(), **case["args"]),
            *O.sample_depthwise_backward(dy.float(), x.float(), r.float(), k.float(), **case["args"]))
    x, r, k, dy = (t.cuda() for t in (x, r, k, dy))
    if shifted:
        x, r, dy = _odd_start(x), _odd_start(r), _odd_start(dy)
    leaves = [t.requires_grad_(True) for t in (x, r, k)]
    y = sample_depthwise(*leaves, **case["args"])
    for name, g, v in zip(("output", "input", "rotation", "weight"), (y.detach(),) + torch.autograd.grad(y, leaves, dy), want):
        assert rel_err(g, v.half()) < 2e-3, name  # hat products, K and products with dy rounded to fp16, the result as well


@pytest.mark.parametrize("n,c,h", [(2, 32, 9), (24, 96, 45), (3, 64, 100), (2, 40, 31)])
@pytest.mark.parametrize("w", [71, 73, 75, 79, 89, 95, 97])
@pytest.mark.parametrize("shifted", [False, True])
def test_forward_and_gradients(n, c, h, w, shifted):
    _check(n, c, h, w, 2, shifted)


@pytest.mark.parametrize("n,c,h,w", [(3, 64, 75, 101), (2, 96, 60, 97), (7, 16, 99, 111), (1, 240, 61, 129)])
@pytest.mark.parametrize("shifted", [False, True])
def test_stride_1(n, c, h, w, shifted):
    """Rows above 96 a warp each: calls that are not small."""
    _check(n, c, h, w, 1, shifted)


@pytest.mark.parametrize("n,c,h,w,stride", [(61, 8, 45, 41, 1), (6, 24, 64, 64, 2), (2, 40, 110, 112, 2), (3, 56, 96, 104, 2), (4, 24, 62, 62, 2), (9, 72, 33, 40, 2)])
def test_calls_between_the_kernels(n, c, h, w, stride):
    """Channels outside a multiple of 16: few of them on odd rows, and grad-input at stride 2 with full, half and no patches at the ends of its rows."""
    _check(n, c, h, w, stride, False)
