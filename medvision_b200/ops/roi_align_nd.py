"""RoIAlign (axis-aligned), 2D and 3D, with autograd.

Same public surface as medvision/ops/roi_align_nd.py: ``RoIAlign2DFunction``,
``RoIAlign3DFunction``, ``roi_align_2d``, ``roi_align_3d`` and the ``RoIAlign`` module
(``RoIAlign(output_size, spatial_scale, sampling_ratio=-1)(features, rois, order=1)``).
"""
import torch.nn as nn

from .. import _C
from ._common import RoiFunction

# features, rois, output_size, spatial_scale, sampling_ratio=0, order=1; differentiable in the features
roi_align_2d = _C._native.roi_align_2d
roi_align_3d = _C._native.roi_align_3d


class RoIAlign2DFunction(RoiFunction):
    ndim, call = 2, staticmethod(roi_align_2d)
    kernels = _C.roi_align_2d_forward, _C.roi_align_2d_backward

    @staticmethod
    def forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio=0, order=1):
        return RoIAlign2DFunction._forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio, order)

    @staticmethod
    def backward(ctx, grad_output):
        return RoIAlign2DFunction._backward(ctx, grad_output)


class RoIAlign3DFunction(RoiFunction):
    ndim, call = 3, staticmethod(roi_align_3d)
    kernels = _C.roi_align_3d_forward, _C.roi_align_3d_backward

    @staticmethod
    def forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio=0, order=1):
        return RoIAlign3DFunction._forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio, order)

    @staticmethod
    def backward(ctx, grad_output):
        return RoIAlign3DFunction._backward(ctx, grad_output)


class RoIAlign(nn.Module):
    """RoI align pooling for axis-aligned proposals.

    features: (N, C, H, W) or (N, C, D, H, W); rois: (n, 5) = (batch_index, x1, y1, x2, y2)
    or (n, 7) = (batch_index, x1, y1, z1, x2, y2, z2), same dtype and device as the features.

    Args:
        output_size (tuple): (h, w) or (d, h, w); its length selects 2D or 3D
        spatial_scale (float): the boxes are multiplied by this number
        sampling_ratio (int): sub-samples per output bin and axis; <= 0 samples adaptively,
            ceil(roi_size / output_size) per axis
    """

    def __init__(self, output_size, spatial_scale, sampling_ratio=-1):
        super().__init__()
        assert iter(output_size)
        self.output_size = output_size
        self.spatial_scale = float(spatial_scale)
        self.sampling_ratio = int(sampling_ratio)
        self.dim = len(self.output_size)
        if self.dim == 2:
            self.roi_align = roi_align_2d
        elif self.dim == 3:
            self.roi_align = roi_align_3d
        else:
            raise Exception("Tried to init RoIAlign module with incorrect output size: {}".format(self.output_size))

    def forward(self, features, rois, order=1):
        assert order in [0, 1], "only support order = 0 (nearest) or 1 (linear)"
        # nearest neighbour takes one sample per bin: averaging samples would blend labels
        sampling_ratio = 1 if order == 0 else self.sampling_ratio
        return self.roi_align(features, rois, self.output_size, self.spatial_scale, sampling_ratio, order)
