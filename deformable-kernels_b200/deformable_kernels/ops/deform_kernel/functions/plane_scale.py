"""Per-(sample, channel) scaling y[n,c] = x[n,c] * k[n,c]: the global deformable kernel's per-sample grouped
convolution (reference modules/deform_kernel.py:105-118) in the 1x1 depthwise case, as one streaming pass with a
fused backward (grad-input and the per-plane reduction grad-k in the same kernel)."""
from ...._native import native

__all__ = ['plane_scale']

plane_scale = native.plane_scale
