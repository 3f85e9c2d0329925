"""The N-d multilinear sampler used by the global deformable kernel, differentiable.

Same name and signature as the reference's functions/nd_linear_sample.py:18-65:
``nd_linear_sample(input[C, s1..sD], coord[B, D]) -> [B, C]``.  The coordinate gradient
is reduced over channels inside the kernel (the reference materialises [B, D, C] and
sums in Python, :49-55) and no ``shape`` tensor is built on the host per call (:22, :36).
"""
from ...._native import native

__all__ = ['nd_linear_sample']

nd_linear_sample = native.nd_linear_sample
