"""The kernels that spread a batch over clusters of blocks: the N-d sampler's array gradient and the fused global kernel."""
import pytest
import torch

from dk_cases import make_nd_case, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.float64: 1e-11, torch.float32: 1e-5, torch.float16: 2e-3}


# one sample; fewer samples than warps; channel remainders; the most and one more cell than 8, 2 and 1 warps' accumulators
# take (96, 384 and 768 cells in fp32); a bank that no accumulator fits
@pytest.mark.parametrize("c,shape,b", [(1, (2, 2), 1), (33, (4, 4), 3), (32, (4, 24), 300), (31, (97,), 200), (65, (16, 24), 129),
                                       (40, (12, 64), 70), (8, (769,), 33), (16, (30, 40), 50)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.float64])
def test_array_gradient(c, shape, b, dtype):
    from deformable_kernels.ops.deform_kernel.functions import nd_linear_sample
    from oracle import dk_oracle as O
    case = make_nd_case(c, shape, b, seed=c + b)
    data, coord, dy = (case[k].to(dtype) for k in ("data", "coord", "grad_output"))
    d, p = data.to(DEV).requires_grad_(True), coord.to(DEV).requires_grad_(True)
    got = torch.autograd.grad(nd_linear_sample(d, p), [d, p], dy.to(DEV))
    up = torch.float32 if dtype == torch.float16 else torch.float64
    want = O.nd_linear_sample_backward(dy.to(up), data.to(up), coord.to(up))
    for a, w in zip(got, want):
        assert rel_err(a, w.to(dtype)) < TOL[dtype]


# channels that leave blocks of a cluster empty, planes of no vector width, a plane too large for one block in the backward
# only, and in both directions
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("n,c,h,w,shape", [(1, 3, 5, 7, (2, 2)), (3, 20, 1, 1, (4, 2)), (2, 72, 9, 13, (3, 3)), (2, 8, 176, 176, (2, 2)),
                                           (1, 16, 300, 200, (2, 3, 2))])
def test_global_kernel(n, c, h, w, shape, dtype):
    from deformable_kernels.modules import GlobalDeformKernel2d
    torch.manual_seed(c)
    m = GlobalDeformKernel2d(shape, c, c, kernel_size=1, groups=c).to(DEV)
    with torch.no_grad():
        m.fc.weight.normal_(0, 0.5)
        m.fc.bias.normal_(0, 0.2)
    x, dy = (torch.randn(n, c, h, w, device=DEV).to(dtype) for _ in range(2))
    params = [m.weight, m.fc.weight, m.fc.bias]
    xi = x.clone().requires_grad_(True)
    assert m._fused_head_ok(xi)
    y = m(xi)
    got = [y.detach()] + list(torch.autograd.grad(y, [xi] + params, dy))
    m._fused_head_ok = lambda _x: False
    m = m.double()
    m._tap_bias = m._tap_bias.double()
    xd = x.double().requires_grad_(True)
    scale = _scale_of(m, xd)
    yd = xd * scale.view(n, c, 1, 1)
    want = [yd.detach()] + list(torch.autograd.grad(yd, [xd, m.weight, m.fc.weight, m.fc.bias], dy.double()))
    for name, a, b in zip(("y", "dx", "dbank", "dfc_weight", "dfc_bias"), got, want):
        assert rel_err(a, b) < (3e-5 if dtype == torch.float32 else 2e-3), "%s: %.3e" % (name, rel_err(a, b))


def _scale_of(m, x):
    """The sampled scale of every (sample, channel) in fp64."""
    from deformable_kernels.ops.deform_kernel.functions import nd_linear_sample
    coord = torch.clamp(m.fc(x.mean((2, 3))) + m._tap_bias, 0, m.weight_shape[0] - 1)
    return nd_linear_sample(m.weight.view(m.out_planes, *m.weight_shape), coord)
