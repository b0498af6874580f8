"""RoIAlignRotated, 2D and 3D, with autograd.

Same public surface as medvision/ops/roi_align_rotated_nd.py: ``RoIAlignRotated2DFunction``,
``RoIAlignRotated3DFunction``, ``roi_align_rotated_2d``, ``roi_align_rotated_3d`` and the
``RoIAlignRotated`` module
(``RoIAlignRotated(output_size, spatial_scale, sampling_ratio=-1, aligned=True)(features, rois, order=1)``).
"""
import torch.nn as nn

from .. import _C
from ._common import RoiFunction

# features, rois, output_size, spatial_scale, sampling_ratio=0, aligned=True, order=1; differentiable in the features
roi_align_rotated_2d = _C._native.roi_align_rotated_2d
roi_align_rotated_3d = _C._native.roi_align_rotated_3d


class RoIAlignRotated2DFunction(RoiFunction):
    ndim, call = 2, staticmethod(roi_align_rotated_2d)
    kernels = _C.roi_align_rotated_2d_forward, _C.roi_align_rotated_2d_backward

    @staticmethod
    def forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio=0, aligned=True, order=1):
        return RoIAlignRotated2DFunction._forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio, aligned, order)

    @staticmethod
    def backward(ctx, grad_output):
        return RoIAlignRotated2DFunction._backward(ctx, grad_output)


class RoIAlignRotated3DFunction(RoiFunction):
    ndim, call = 3, staticmethod(roi_align_rotated_3d)
    kernels = _C.roi_align_rotated_3d_forward, _C.roi_align_rotated_3d_backward

    @staticmethod
    def forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio=0, aligned=True, order=1):
        return RoIAlignRotated3DFunction._forward(ctx, features, rois, output_size, spatial_scale, sampling_ratio, aligned, order)

    @staticmethod
    def backward(ctx, grad_output):
        return RoIAlignRotated3DFunction._backward(ctx, grad_output)


class RoIAlignRotated(nn.Module):
    """RoI align pooling for rotated proposals.

    features: (N, C, H, W) or (N, C, D, H, W); rois: (n, 6) =
    (batch_index, center_x, center_y, w, h, angle) or (n, 10) =
    (batch_index, center_x, center_y, center_z, w, h, d, angle_x, angle_y, angle_z), angles in
    radians, same dtype and device as the features.  In 3D the sample lattice of the roi is
    rotated by Rz(angle_z) * Ry(angle_y) * Rx(angle_x) about the roi centre.

    Args:
        output_size (tuple): (h, w) or (d, h, w); its length selects 2D or 3D
        spatial_scale (float): centre and size are multiplied by this number
        sampling_ratio (int): sub-samples per output bin and axis; <= 0 samples adaptively
        aligned (bool): True shifts the scaled centre by -0.5 so that pixel centres sit at
            half-integer continuous coordinates (the detectron2 convention) and does not clamp
            the roi size; False keeps the legacy convention and forces sizes to >= 1
    """

    def __init__(self, output_size, spatial_scale, sampling_ratio=-1, aligned=True):
        super().__init__()
        assert iter(output_size)
        self.output_size = output_size
        self.spatial_scale = float(spatial_scale)
        self.sampling_ratio = int(sampling_ratio)
        self.aligned = aligned
        self.dim = len(self.output_size)
        if self.dim == 2:
            self.roi_align = roi_align_rotated_2d
        elif self.dim == 3:
            self.roi_align = roi_align_rotated_3d
        else:
            raise Exception("Tried to init RoIAlign module with incorrect output size: {}".format(self.output_size))

    def forward(self, features, rois, order=1):
        assert order in [0, 1], "only support order = 0 (nearest) or 1 (linear)"
        sampling_ratio = 1 if order == 0 else self.sampling_ratio
        return self.roi_align(features, rois, self.output_size, self.spatial_scale, sampling_ratio,
                              self.aligned, order)
