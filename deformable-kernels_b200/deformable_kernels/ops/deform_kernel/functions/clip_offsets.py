"""Clipping and scaling of produced offsets in one pass (reference modules/deform_kernel.py:185-218 `_clip_rotation`,
:165-170 `rotation * weight_dilate`, :273-276 offset clamp and `* dilation`):

    v = offsets * dilate + bias[channel];  output = (clamp(v, lo, hi) - bias[channel]) / dilate * post_scale
"""
from ...._native import native

__all__ = ['clip_offsets']


def clip_offsets(offsets, bias=None, lo=float('-inf'), hi=float('inf'), dilate=1.0, post_scale=1.0):
    return native.clip_offsets(offsets, bias, lo, hi, dilate, post_scale)
