"""Offset and bank gradients of the local operator from bf16 pieces of fp32 values: calls of 64 tiles and more, with channels that do not fill a step of 8 or a
chunk of 32, tiles of odd shapes, pixels that do not fill a warp, both strides, and values that are not finite."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(case, dtype):
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    x, r, w, dy = (case[k].to(dtype).to(DEV) for k in ("input", "rotation", "weight", "grad_output"))
    for t in (r, w):
        t.requires_grad_(True)
    return torch.autograd.grad(sample_depthwise(x, r, w, **case["args"]), [r, w], dy)


def _want(case, dtype):
    from oracle import dk_oracle as O
    a = [case[k].to(dtype).double() for k in ("grad_output", "input", "rotation", "weight")]
    return O.sample_depthwise_backward(*a, **case["args"])[1:]


@pytest.mark.parametrize("n,c,h,w,stride,scope", [
    (70, 3, 5, 5, 1, (4, 4)), (66, 8, 12, 8, 1, (4, 4)), (64, 33, 1, 7, 1, (4, 4)), (9, 40, 25, 31, 1, (3, 3)), (3, 72, 40, 57, 1, (4, 4)),
    (2, 104, 96, 50, 1, (2, 4)), (65, 136, 4, 3, 1, (1, 4)), (4, 24, 8, 200, 1, (4, 1)), (64, 8, 16, 17, 2, (4, 4)), (5, 56, 60, 61, 2, (4, 4)),
    (70, 200, 14, 13, 2, (3, 4)),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_shapes(n, c, h, w, stride, scope, dtype):
    case = make_case(n, c, h, w, scope=scope, stride=stride, rot_std=1.0, seed=c + w)
    for name, g, v in zip(("rotation", "weight"), _run(case, dtype), _want(case, dtype)):
        assert rel_err(g, v.to(dtype)) < (1e-5 if dtype == torch.float32 else 2e-3), name


@pytest.mark.parametrize("n,c,h,w,stride", [(8, 64, 56, 56, 1), (40, 96, 30, 41, 2), (64, 384, 14, 14, 1)])
def test_error_against_fp64(n, c, h, w, stride):
    """2-norm of fp32 results.  Pieces: 2^-26 of a product in the mean; the products of a step are truncated at 2^-23 of their sum, 6e-8 in the mean; the
    coordinate is rounded at its size for the hat products (1.2e-7 of a kernel value, bank only); rounded additions of C / 16 steps
    (offsets) or of the pixels' steps (bank), 8.6e-8 sqrt(L / 24) for chains of L = C / 16 and of 12 steps a tile: 1.2e-7 and 2.6e-7."""
    case = make_case(n, c, h, w, stride=stride, rot_std=1.0, seed=c)
    for name, g, v, bound in zip(("rotation", "weight"), _run(case, torch.float32), _want(case, torch.float32), (1.7e-7, 2.9e-7)):
        err = float((g.double().cpu() - v).norm() / v.norm())
        assert err < bound, "%s %.3e" % (name, err)


def test_products_that_are_not_finite():
    """An infinite dy reaches the offsets of its own pixel and the bank cells its taps sample, in its own channel."""
    case = make_case(16, 40, 20, 24, rot_std=0.4, seed=4)
    plain = _run(case, torch.float32)
    case["grad_output"][5, 17, 9, 11] = float("inf")
    got = _run(case, torch.float32)
    other = torch.ones_like(got[0], dtype=torch.bool)
    other[5, :, 9, 11] = False
    torch.testing.assert_close(got[0][other], plain[0][other], rtol=1e-5, atol=1e-5)
    assert not torch.isfinite(got[0][5, :, 9, 11]).all()
    changed = ~torch.isfinite(got[1])
    assert 0 < int(changed[17].sum()) and int(changed.sum()) == int(changed[17].sum())
    u = torch.zeros(4, 4, dtype=torch.bool)  # cells that the nine taps of the pixel touch
    rot = case["rotation"][5, :, 9, 11].view(9, 2)
    for t in range(9):
        a, b = int(torch.floor(t // 3 + rot[t, 0] + 0.5)), int(torch.floor(t % 3 + rot[t, 1] + 0.5))
        for i in (a, a + 1):
            for j in (b, b + 1):
                if 0 <= i < 4 and 0 <= j < 4:
                    u[i, j] = True
    assert not changed[17, 0][~u.to(DEV)].any()


@pytest.mark.parametrize("n,c,h,w,stride", [(16, 16, 61, 63, 2), (27, 16, 11, 17, 1), (5, 40, 80, 86, 2), (4, 120, 53, 57, 1), (8, 200, 30, 28, 1)])
def test_no_less_exact_than_each_gradient_alone(n, c, h, w, stride):
    """Either gradient alone comes from a kernel with an fp32 multiply-add per term; how many are wanted must not cost precision."""
    from deformable_kernels.ops.deform_kernel.functions import sample_depthwise
    case = make_case(n, c, h, w, stride=stride, rot_std=1.0, seed=c + h)
    both, want = _run(case, torch.float32), _want(case, torch.float32)
    x, r, k, dy = (case[name].to(DEV) for name in ("input", "rotation", "weight", "grad_output"))
    for i, (name, leaf) in enumerate((("rotation", r), ("weight", k))):
        leaf.requires_grad_(True)
        alone, = torch.autograd.grad(sample_depthwise(x, r, k, **case["args"]), leaf, dy)
        leaf.requires_grad_(False)
        error = [float((g.double().cpu() - want[i]).norm()) for g in (both[i], alone)]
        assert error[0] < 1.01 * error[1], "%s %.3e %.3e" % (name, *error)  # a 2-norm over 2e4 elements and more: 1 % is its own scatter


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["weight", "grad_output", "input", "both"])
def test_where_the_offset_gradients_are_not_finite(where, value, dtype):
    """Exactly where the oracle's are not: a value of the bank reaches the samples of its cell, one of dy or x those of its pixel."""
    case = make_case(16, 40, 20, 24, rot_std=0.8, seed=6)
    if where in ("weight", "both"):
        case["weight"][11, 0, 1, 2] = case["weight"][39, 0, 3, 0] = value
    if where in ("grad_output", "both"):
        case["grad_output"][3, 17, 9, 11] = case["grad_output"][7, 2, 19, 23] = value
    if where in ("input", "both"):
        case["input"][2, 5, 0, 7] = case["input"][15, 39, 13, 23] = value
    (got, dw), (want, dw_want) = _run(case, dtype), _want(case, dtype)
    finite = torch.isfinite(want)
    assert (~finite).any() and finite.any()
    assert torch.equal(torch.isfinite(got).cpu(), finite)
    assert rel_err(got.cpu()[finite], want[finite].to(dtype)) < (1e-5 if dtype == torch.float32 else 2e-3)
    assert torch.isfinite(dw).cpu()[torch.isfinite(dw_want)].all()


def test_an_infinite_bank_value_gives_infinities():
    """Its sign and that of dy * x decide, as with a multiply-add per term: not the NaN of the pieces of infinity."""
    case = make_case(16, 40, 20, 24, rot_std=0.8, seed=6)
    case["weight"][11, 0, 1, 2] = float("inf")
    got, want = _run(case, torch.float32)[0].double().cpu(), _want(case, torch.float32)[0]
    assert torch.isinf(want).any() and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
