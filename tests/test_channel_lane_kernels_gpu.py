"""The local operator with any number of channels, against the CPU oracle: fp32 runs on the tcgen05 kernels (one channel per
TMEM lane), fp16 there on wide rows, else on the mma.sync kernels with a partly filled last slab of channels.  The sizes are the edges of their tiles:
32-channel groups (1 to 5 of them, full and partial, so that every
placement of the remaining groups on the lanes occurs), 8-pixel segments, rows with and without TMA, planes of one row or one
pixel, steps that span samples, more channels than one block takes."""
import pytest
import torch

from dk_cases import make_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [
    (1, 8, 1, 1), (5, 16, 1, 9), (3, 24, 7, 7), (2, 32, 8, 8), (2, 40, 9, 16), (1, 56, 17, 24), (2, 72, 19, 23),
    (1, 104, 12, 33), (2, 136, 5, 40), (1, 160, 28, 28), (1, 200, 14, 14), (1, 264, 3, 64), (9, 280, 4, 4), (1, 1096, 6, 10),
    (1, 24, 112, 112), (1, 8, 2, 200), (1, 32, 110, 110), (2, 48, 31, 57),
    (2, 72, 31, 48), (5, 264, 2, 32),
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
