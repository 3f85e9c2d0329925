"""GlobalDeformKernel2d with a 1x1 depthwise kernel as one forward and one backward call
(reference modules/deform_kernel.py:76-118: global average pool -> linear coordinate head ->
clamp -> N-d linear sample of the bank -> per-sample grouped convolution, here a per-plane
scale): ``global_dk_scale(input, bank, fc_weight, fc_bias, tap_bias)``, the bank as
[C, shape...] or, as the layer stores it, [C, 1, shape...].  The coordinate head runs in
fp32 whatever the dtype of the feature map."""
from ...._native import native

__all__ = ['global_dk_scale']

global_dk_scale = native.global_dk_scale
