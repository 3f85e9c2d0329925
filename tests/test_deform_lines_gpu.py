"""DK + DCN in fp16 with the operands in channel order: units of 64 channels, strips of 16 columns, windows of 8 columns and groups of 16
pixels or samples, each with remainders, against the fp32 oracle (grad-input also bit for bit against itself)."""
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "deformable-kernels_b200"))
sys.path.insert(0, ROOT)

from dk_cases import make_case, rel_err  # noqa: E402

pytestmark = pytest.mark.gpu
NAMES = ("grad_input", "grad_offset", "grad_rotation", "grad_weight")


def _run(case, rotation=True):
    from deformable_kernels.ops.deform_kernel.functions import deform_sample_depthwise
    dy, x, o, r, w = (case[k].to(torch.float16).cuda() for k in ("grad_output", "input", "offset", "rotation", "weight"))
    leaves = [t.requires_grad_(True) for t in ((x, o, r, w) if rotation else (x, o, w))]
    y = deform_sample_depthwise(x, o, r if rotation else None, w, **case["args"])
    names = NAMES if rotation else tuple(n for n in NAMES if n != "grad_rotation")
    return dict(zip(("output",) + names, (y.detach(),) + torch.autograd.grad(y, leaves, dy)))


def _want(case):
    from oracle import dk_oracle as O
    dy, x, o, r, w = (case[k].to(torch.float16).float() for k in ("grad_output", "input", "offset", "rotation", "weight"))
    return dict(zip(("output",) + NAMES, (O.deform_sample_depthwise_forward(x, o, r, w, **case["args"]),) +
                    tuple(O.deform_sample_depthwise_backward(dy, x, o, r, w, **case["args"]))))


def _check(case, rotation=True):
    if not rotation:
        case["rotation"] = torch.zeros_like(case["rotation"])
    got, want = _run(case, rotation), _want(case)
    for k, v in got.items():
        # corner weights, hat products, K and the products with dy rounded to fp16 (2^-11 each), the result as well
        assert rel_err(v, want[k].half()) < 2e-3, k
    return got


@pytest.mark.parametrize("n,c,h,w,stride,scope,rotation", [
    (32, 48, 17, 16, 1, (4, 4), True),     # part of a unit; a strip without remainder
    (40, 64, 18, 34, 2, (4, 4), True),     # one unit, four groups of pixels per block; columns of y 17
    (12, 144, 20, 20, 1, (3, 3), True),    # three units: a block of three warps
    (7, 320, 16, 36, 1, (4, 4), True),     # five units: two sets of channels; strips 16, 16, 4
    (6, 272, 25, 30, 2, (2, 4), True),     # odd rows of y, even columns of x
    (20, 128, 9, 50, 1, (3, 3), False),    # no kernel-space offsets
    (50, 64, 3, 200, 1, (1, 4), True),     # fewer rows than a band
    (3, 960, 21, 15, 1, (4, 4), True),     # four sets; odd columns
    (24, 96, 56, 6, 1, (4, 1), True),      # narrower than a window
])
def test_shapes(n, c, h, w, stride, scope, rotation):
    case = make_case(n, c, h, w, scope=scope, stride=stride, rot_std=0.7, off_std=2.0, seed=7)
    _check(case, rotation)


def test_offsets_that_collapse_and_leave():
    """Every tap of a sample on one point (one cell holds all records, far more than a chunk), and points far outside, infinite or NaN."""
    case = make_case(10, 160, 14, 18, scope=(4, 4), rot_std=0.5, off_std=1.0, seed=8)
    off = case["offset"].view(10, 9, 2, 14, 18)
    rows, cols = torch.arange(14.).view(1, 14, 1), torch.arange(18.).view(1, 1, 18)
    for t in range(9):
        off[0, t, 0], off[0, t, 1] = 6.25 - (rows[0] - 1 + t // 3), 7.5 - (cols[0] - 1 + t % 3)
    off[1] = 1e4
    off[2, :, 0, 3, 4], off[2, :, 1, 5, 6], off[2, 4, 0, 7, 7] = float("nan"), float("inf"), -float("inf")
    got = _check(case)
    assert torch.equal(got["grad_input"][1], torch.zeros_like(got["grad_input"][1]))


def test_grad_input_is_the_same_in_every_run():
    case = make_case(16, 96, 31, 28, scope=(4, 4), rot_std=0.5, off_std=2.0, seed=9)
    first = _run(case)["grad_input"]
    for _ in range(3):
        assert torch.equal(first, _run(case)["grad_input"])


def test_values_that_are_not_finite_stay_with_their_samples():
    """An infinite dy reaches the pixels its taps touch in its own channel; the rest of grad-input keeps its value."""
    case = make_case(8, 192, 20, 24, scope=(4, 4), rot_std=0.3, off_std=1.0, seed=10)
    plain = _run(case)["grad_input"]
    case["grad_output"][3, 100, 9, 11] = float("inf")
    got = _run(case)["grad_input"]
    changed = ~torch.isfinite(got)
    assert 4 <= int(changed.sum()) <= 36 and bool(changed[3, 100].any()) and int(changed.sum()) == int(changed[3, 100].sum())
    # a window with such a value is summed pixel by pixel in fp32, not in pieces of 22 bits
    torch.testing.assert_close(got[~changed], plain[~changed], rtol=2e-3, atol=2e-3)


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_bank_values_that_are_not_finite_stay_in_their_channel(value):
    """K of a channel comes out of the same products as that of the channel 32 away."""
    case = make_case(8, 192, 20, 24, scope=(4, 4), rot_std=0.3, off_std=1.0, seed=11)
    plain = _run(case)
    for c in (5, 70, 127):
        case["weight"][c, 0, 1, 2] = value
    got = _run(case)
    rest = [c for c in range(192) if c not in (5, 70, 127)]
    for k in ("output", "grad_input"):
        torch.testing.assert_close(got[k][:, rest], plain[k][:, rest], rtol=2e-3, atol=2e-3)
        assert all(not torch.isfinite(got[k][:, c]).all() for c in (5, 70, 127)), k
    assert torch.equal(got["grad_weight"], plain["grad_weight"])  # does not depend on the bank


@pytest.mark.parametrize("rotation", [True, False])
def test_forward_without_its_scratch(rotation):
    """The kernels with planes on chip take the same calls: no scratch, or too little, is not an error."""
    from deformable_kernels import _cabi as C
    case = make_case(6, 128, 28, 30, scope=(4, 4) if rotation else (3, 3), rot_std=0.5, off_std=1.0, seed=12)
    want = _run(case, rotation)["output"]
    x, o, r, w = (case[k].to(torch.float16).cuda() for k in ("input", "offset", "rotation", "weight"))
    g = C.geom(tuple(x.shape), (3, 3), (1, 1), (1, 1), (1, 1), tuple(w.shape[2:]), 1)
    need = C.lib.dk_deform_sample_depthwise_forward_workspace_bytes(g, C.DK_F16)
    assert need > 0
    for size in (0, 256, need - 256, need):
        ws, y = torch.empty(max(size, 1), dtype=torch.uint8, device="cuda"), torch.empty_like(want)
        status = C.lib.dk_deform_sample_depthwise_forward_ws(C.ptr(x), C.ptr(o), C.ptr(r if rotation else None), C.ptr(w), C.ptr(y), g, C.DK_F16,
                                                             C.ptr(ws if size else None), size, C.stream_ptr(x.device))
        assert status == 0, size
        assert rel_err(y, want) < 2e-3, size  # both round corner weights, hat products and K to fp16


@pytest.mark.parametrize("top,mean", [(800, 70), (1600, 30)])
def test_offset_gradients_where_only_the_corners_are_large(top, mean):
    """|dy K x| beyond fp16 with |dy x| and |dy K dx| inside it: a scaled loss and an input far from zero.  The differences of the corners are exact."""
    case = make_case(32, 64, 30, 28, scope=(4, 4), rot_std=0.7, off_std=2.0, seed=13)
    case["grad_output"] = case["grad_output"].clamp(-1, 1) * top
    case["input"] = mean + case["input"]
    case["weight"] *= 3.0
    assert top * case["input"].abs().max() < 65504 < top * mean * case["weight"].abs().max() * 0.75
    got, want = _run(case)["grad_offset"].cpu(), _want(case)["grad_offset"]
    # samples whose four corners lie in the image: beside it the difference is the value itself
    off = case["offset"].half().float().view(32, 9, 2, 30, 28)
    tap = torch.arange(9.).view(9, 1, 1)
    h, w = off[:, :, 0] + torch.arange(30.).view(30, 1) - 1 + tap // 3, off[:, :, 1] + torch.arange(28.) - 1 + tap % 3
    inside = ((h >= 0) & (h < 29) & (w >= 0) & (w < 27)).repeat_interleave(2, 1)
    got, want = got[inside], want[inside]
    assert want.abs().max() < 65504 and torch.isfinite(got).all()
    assert rel_err(got, want.half()) < 2e-3


@pytest.mark.parametrize("n,c,h,w,stride", [(8, 192, 20, 24, 1), (6, 272, 25, 30, 2), (4, 144, 26, 29, 1)])
def test_grad_input_of_values_that_are_not_finite(n, c, h, w, stride):
    """Not finite exactly where the oracle is not: channels of every lane and half, both columns of a pair, windows with a remainder."""
    case = make_case(n, c, h, w, scope=(4, 4), stride=stride, rot_std=0.3, off_std=1.5, seed=w)
    gen = torch.Generator().manual_seed(5)
    dy = case["grad_output"]
    for k in range(40):
        at = [int(torch.randint(s, (1,), generator=gen)) for s in dy.shape]
        dy[at[0] // 2, at[1], at[2], at[3]] = (float("inf"), -float("inf"), float("nan"))[k % 3]
    case["weight"][c - 3, 0, 1, 1], case["weight"][36, 0, 2, 0] = float("inf"), float("nan")
    got, want = _run(case)["grad_input"].cpu(), _want(case)["grad_input"]
    finite = torch.isfinite(want)
    assert 100 < int((~finite).sum()) < finite.numel() // 10
    assert torch.equal(torch.isfinite(got), finite)
    assert rel_err(got[finite], want[finite].half()) < 2e-3


def _behind(t, halves):
    """The same values so many halves behind an aligned address."""
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    return buf[halves:halves + t.numel()].view(t.shape).copy_(t)


@pytest.mark.parametrize("n,c,h,w,stride", [(8, 64, 24, 40, 1), (24, 64, 24, 40, 1), (40, 48, 32, 60, 2)])  # forward of the first: planes on chip
@pytest.mark.parametrize("halves", [1, 2, 4])
def test_operands_at_any_address(n, c, h, w, stride, halves):
    """Widths and planes allow the wide loads and stores, the addresses do not: the results are the same, of most kernels bit for bit."""
    from deformable_kernels import _cabi as C
    case = make_case(n, c, h, w, scope=(4, 4), stride=stride, rot_std=0.7, off_std=2.0, seed=14)
    dy, x, o, r, wt = (case[k].to(torch.float16).cuda() for k in ("grad_output", "input", "offset", "rotation", "weight"))
    g = C.geom(tuple(x.shape), (3, 3), (stride, stride), (1, 1), (1, 1), (4, 4), 1)
    size = max(C.lib.dk_deform_sample_depthwise_forward_workspace_bytes(g, C.DK_F16), C.lib.dk_deform_sample_depthwise_backward_workspace_bytes(g, C.DK_F16))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    s = C.stream_ptr(x.device)
    results = []
    for k in (0, halves):
        a, b, d, e, f = (_behind(t, k) for t in (dy, x, o, r, wt))
        y, dx, do, dr, dw = (_behind(torch.zeros_like(t), k) for t in (dy, x, o, r, wt))
        assert C.lib.dk_deform_sample_depthwise_forward_ws(C.ptr(b), C.ptr(d), C.ptr(e), C.ptr(f), C.ptr(y), g, C.DK_F16, C.ptr(ws), size, s) == 0
        assert C.lib.dk_deform_sample_depthwise_backward(C.ptr(a), C.ptr(b), C.ptr(d), C.ptr(e), C.ptr(f), C.ptr(dx), C.ptr(do), C.ptr(dr), C.ptr(dw), g,
                                                         C.DK_F16, C.ptr(ws), size, s) == 0
        results.append([t.clone() for t in (y, dx, do, dr, dw)])
    for k, (first, other) in enumerate(zip(*results)):
        if n > 8 or k == 0:
            assert torch.equal(first, other)
        else:  # the kernels of few samples add in the order of the day: two roundings to fp16
            assert rel_err(first, other) < 1e-3


def test_scratch_at_any_word():
    """Lines want 16 bytes; scratch that begins between them is left to the kernels that take it."""
    from deformable_kernels import _cabi as C
    case = make_case(24, 64, 24, 40, scope=(4, 4), rot_std=0.7, off_std=2.0, seed=14)
    dy, x, o, r, w = (case[k].to(torch.float16).cuda() for k in ("grad_output", "input", "offset", "rotation", "weight"))
    g = C.geom(tuple(x.shape), (3, 3), (1, 1), (1, 1), (1, 1), (4, 4), 1)
    size = max(C.lib.dk_deform_sample_depthwise_forward_workspace_bytes(g, C.DK_F16), C.lib.dk_deform_sample_depthwise_backward_workspace_bytes(g, C.DK_F16))
    s, want = C.stream_ptr(x.device), _want(case)
    ws = torch.empty(size // 4 + 4, dtype=torch.float32, device="cuda")[1:]
    got = [torch.empty_like(t) for t in (x, x, o, r, w)]
    assert C.lib.dk_deform_sample_depthwise_forward_ws(*(C.ptr(t) for t in (x, o, r, w, got[0])), g, C.DK_F16, C.ptr(ws), size, s) == 0
    assert C.lib.dk_deform_sample_depthwise_backward(*(C.ptr(t) for t in (dy, x, o, r, w, *got[1:])), g, C.DK_F16, C.ptr(ws), size, s) == 0
    for k, v in zip(("output",) + NAMES, got):
        assert rel_err(v, want[k].half()) < 2e-3, k
