"""The local deformable kernel and DK + DCN as differentiable functions.

Same names, argument order and defaults as the reference's
functions/filter_sample_depthwise.py:18-211 (``sample_depthwise``,
``deform_sample_depthwise``); what differs underneath (csrc/dk_torch.cpp):
  * one fused C-ABI call computes every requested gradient (the reference issues three
    or four launches and zero-fills each buffer first, :63-85 and :151-189);
  * the backward returns one gradient per forward argument (the reference returns one
    too few, :87 and :191, which current PyTorch rejects);
  * work is enqueued on the current stream of the input's device;
  * offsets and banks that differ in dtype from the activations (offsets produced under
    autocast, fp32 parameters) follow the input's dtype.
CPU tensors raise NotImplementedError exactly as in the reference (:43-44).
"""
from ...._native import native

__all__ = ['sample_depthwise', 'deform_sample_depthwise']


def sample_depthwise(input, rotation, weight, kernel_size=(3, 3), stride=(1, 1), padding=(1, 1), dilation=(1, 1),
                     rotation_groups=1):
    return native.sample_depthwise(input, rotation, weight, kernel_size, stride, padding, dilation, rotation_groups, True)


def deform_sample_depthwise(input, offset, rotation, weight, kernel_size=(3, 3), stride=(1, 1), padding=(1, 1),
                            dilation=(1, 1), rotation_groups=1):
    return native.deform_sample_depthwise(input, offset, rotation, weight, kernel_size, stride, padding, dilation,
                                          rotation_groups, True)


class SampleDepthwiseFunction:
    """The operator with one dtype per call: mixed dtypes raise TypeError."""

    @staticmethod
    def apply(input, rotation, weight, kernel_size=(3, 3), stride=(1, 1), padding=(1, 1), dilation=(1, 1),
              rotation_groups=1):
        return native.sample_depthwise(input, rotation, weight, kernel_size, stride, padding, dilation, rotation_groups, False)


class DeformableSampleDepthwiseFunction:
    """The operator with one dtype per call: mixed dtypes raise TypeError."""

    @staticmethod
    def apply(input, offset, rotation, weight, kernel_size=(3, 3), stride=(1, 1), padding=(1, 1), dilation=(1, 1),
              rotation_groups=1):
        return native.deform_sample_depthwise(input, offset, rotation, weight, kernel_size, stride, padding, dilation,
                                              rotation_groups, False)
