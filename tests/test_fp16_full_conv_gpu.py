"""fp16 with channels that are no multiple of 16: forward and grad-input with fp32 kernel values from mma.sync.  Parts of a 16-channel slab, rows
that lie end to end (even) and padded (odd), single rows and columns, scopes of up to 16 cells; nothing but the result is rounded to fp16;
values that are not finite stay with the samples that touch them."""
import pytest
import torch

from dk_cases import make_case

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(case):
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    x, r, w, dy = (case[k].half().to(DEV) for k in ("input", "rotation", "weight", "grad_output"))
    x.requires_grad_(True)
    y = sample_depthwise(x, r, w, **case["args"])
    return y.detach(), torch.autograd.grad(y, x, dy)[0]


def _want(case):
    from oracle import dk_oracle as O
    a = {k: case[k].half().double() for k in ("input", "rotation", "weight", "grad_output")}
    return (O.sample_depthwise_forward(a["input"], a["rotation"], a["weight"], **case["args"]),
            O.sample_depthwise_backward(a["grad_output"], a["input"], a["rotation"], a["weight"], **case["args"])[0])


@pytest.mark.parametrize("n,c,h,w,scope", [(2, 1, 9, 10, (4, 4)), (3, 8, 7, 7, (4, 4)), (2, 24, 20, 22, (4, 4)), (1, 72, 13, 101, (4, 4)),
                                           (2, 40, 1, 18, (3, 5)), (2, 13, 30, 1, (2, 8)), (1, 200, 6, 54, (3, 3)), (40, 56, 14, 14, (4, 4)),
                                           (1, 104, 33, 6, (1, 4)), (2, 8, 5, 150, (4, 4))])
@pytest.mark.parametrize("stride", [1, 2])
def test_only_the_result_is_rounded(n, c, h, w, scope, stride):
    """Rounding to fp16 is off by up to 2^-11 of a value, 2^-11 / sqrt(6) = 2.0e-4 in the mean over a binade at the most."""
    case = make_case(n, c, h, w, scope=scope, stride=stride, rot_std=0.8, seed=c + w)
    for g, v in zip(_run(case), _want(case)):
        got, rounded = g.double().cpu(), v.half().double()
        assert float((got - v).norm()) < 1.02 * float((rounded - v).norm()) + 1e-6 * float(v.norm())


@pytest.mark.parametrize("stride", [1, 2])
def test_small_hat_products_keep_their_bits(stride):
    """Kernel values that come from the far edge of a hat alone.  Fractions of 2^-22 and 2^-10 keep every coordinate exact, so only the rounding
    of the result is left; their products have up to 20 bits, the last of them 2^-32."""
    case = make_case(2, 24, 14, 18, scope=(3, 5), stride=stride, seed=3)
    rot = case["rotation"]
    g = torch.Generator().manual_seed(4)
    rot[:, 0::2] = torch.randint(-900, 900, rot[:, 0::2].shape, generator=g).to(rot.dtype) * 2.0 ** -10
    rot[:, 1::2] = torch.randint(40, 400, rot[:, 1::2].shape, generator=g).to(rot.dtype) * 2.0 ** -22
    case["weight"][..., :4] = 0
    case["weight"][..., 4] *= 1000  # the last column of cells: taps of the last column, a fraction beyond the cell beside it
    for got, v in zip(_run(case), _want(case)):
        got, rounded = got.double().cpu(), v.half().double()
        assert float((got - v).norm()) < 1.02 * float((rounded - v).norm()) + 1e-6 * float(v.norm())


@pytest.mark.parametrize("w,stride", [(22, 1), (26, 2), (21, 1), (23, 2)])
def test_values_that_are_not_finite(w, stride):
    case = make_case(2, 24, 10, w, stride=stride, rot_std=0.4, seed=w)
    plain = _run(case)
    case["input"][1, 5, 4, 0] = float("inf")
    case["grad_output"][0, 7, 2, -1] = float("nan")
    got = _run(case)
    far = torch.ones_like(got[0][1, 5], dtype=torch.bool)
    far[:, :2] = False
    assert not torch.isfinite(got[0][1, 5]).all() and torch.equal(got[0][1, 5][far], plain[0][1, 5][far])
    assert torch.equal(got[0][0], plain[0][0]) and torch.equal(got[0][1, 6:], plain[0][1, 6:])
    far = torch.ones_like(got[1][0, 7], dtype=torch.bool)
    far[:, -4:] = False
    assert torch.isnan(got[1][0, 7]).any() and torch.equal(got[1][0, 7][far], plain[1][0, 7][far]) and torch.equal(got[1][1], plain[1][1])
    case = make_case(2, 24, 10, w, stride=stride, rot_std=0.4, seed=w)
    case["weight"][9, 0, 3, 3] = float("inf")  # touched by few samples
    got = _run(case)
    for g, p in zip(got, plain):
        keep = torch.isfinite(g[:, 9])
        assert 0 < int(keep.sum()) < keep.numel()
        torch.testing.assert_close(g[:, 9][keep], p[:, 9][keep], rtol=2e-3, atol=1e-3)
        rest = [c for c in range(24) if c != 9]
        torch.testing.assert_close(g[:, rest], p[:, rest], rtol=2e-3, atol=1e-3)
