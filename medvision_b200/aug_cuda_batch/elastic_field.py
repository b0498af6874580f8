"""What the batched and the single-sample elastic deformation share: the draw of the coarse grid of control points, the dense
displacement field, and the warp of a call's fields.

The fields are warped straight from the coarse grid (``mvr_elastic``): a voxel's displacement is formed where it is used, and
the dense field -- 12 bytes per voxel that would be written once and read per field -- exists only when it is asked for
(``dense_field`` / ``tmp_params``).  Coarse grids the kernel has no room for, other interpolation orders and other element
types take the two-step form: one ``affine_*`` blow-up, one ``apply_offset_*`` per field."""
import numpy as np
import torch

from .base import global_bit_generator, overrides
from .. import _C
from ..ops.cuda_fun_tools import affine_2d, affine_3d, apply_offset_2d, apply_offset_3d


class ElasticField:
    """Mixin; the class provides ``dim``, ``image_shape``, ``img_type``, ``num_control_points``, ``max_displacement``,
    ``num_locked_borders``, ``params`` and ``_field_order`` (interpolation of the blow-up)."""
    _transform = None  # the transform itself, which a subclass may override
    _dense = None    # the dense field, once it has been asked for
    _device = None   # where the fields of the current parameters were warped

    @property
    def tmp_params(self):
        if self._dense is None and self._device is not None and self.params is not None:
            self._dense = self._blow_up(self._device)
        return self._dense

    @tmp_params.setter
    def tmp_params(self, value):
        self._dense, self._device = value, None

    def _draw_coarse(self, *batch):
        """Coarse displacements (*batch, *grid, dim), at most ``max_displacement`` half grid cells, the outermost
        ``num_locked_borders`` control points of every axis zero."""
        grid = self.to_tuple(self.num_control_points, self.dim)
        reach = self.max_displacement * (np.array(self.image_shape) / (np.array(grid) - 1)) / 2
        coarse = np.empty((*batch, *grid, self.dim), dtype=np.float32)
        generator = global_bit_generator()
        with generator.lock:  # 2 * rand(*grid, dim).astype(float32) - 1 per sample, in [-1, 1)
            _C._native.draw_coarse(generator.capsule, batch[0] if batch else 1, grid, reach.astype(np.float32),
                                   self.num_locked_borders, coarse)
        return coarse

    def _batched_params(self):
        """The parameters as (B, *grid, dim)."""
        return self.params if self.params.ndim == self.dim + 2 else self.params[None]

    def _coarse_tensor(self):
        return torch.from_numpy(np.ascontiguousarray(self._batched_params(), dtype=np.float32))

    def _blow_up(self, device):
        """(B, dim, *image_shape) float32 on ``device``."""
        shape = tuple(self.image_shape)
        if self._field_order == 3:
            field = _C._native.elastic(self._coarse_tensor(), self.num_locked_borders, shape, torch.empty(0, device=device), None,
                                       None)
            if field is not None:
                return field
        coarse = self._coarse_tensor().permute(0, self.dim + 1, *range(1, self.dim + 1)) / 2  # channels first; halved to smooth
        grid = coarse.shape[2:]
        rois = np.zeros((len(coarse), 2 * self.dim + (2 if self.dim == 2 else 4)), dtype=np.float32)
        rois[:, 0] = np.arange(len(coarse))
        rois[:, 1:1 + self.dim] = [i / 2 for i in grid[::-1]]
        rois[:, 1 + self.dim:1 + 2 * self.dim] = [i - (2 * self.num_locked_borders - 1) for i in grid[::-1]]
        fn = affine_2d if self.dim == 2 else affine_3d
        return fn(coarse.contiguous().to(device), torch.from_numpy(rois).to(device), shape, 1, 1, True, self._field_order)

    def _warp_with_dense_field(self, image, field, order):
        """image (B, C, *image_shape) by the dense field; labels (order 0) through the image type, as int32."""
        if order == 0:
            image = image.to(self.img_type)
        image = (apply_offset_2d if self.dim == 2 else apply_offset_3d)(image, field, order=order)
        return image.int() if order == 0 else image

    def _warp_coarse(self, images, labels):
        """The fields (B, C, *image_shape) straight from the coarse grid; None where that takes the two-step form."""
        fields = images + labels
        if self._field_order != 3 or self._dense is not None or not fields or not all(t.is_cuda for t in fields):
            return None
        device = fields[0].device
        like = images[0] if images and images[0].dtype == self.img_type else torch.empty(0, dtype=self.img_type, device=device)
        both = _C._native.elastic(self._coarse_tensor(), self.num_locked_borders, tuple(self.image_shape), like, images, labels)
        if both is not None:
            self._device = device
        return both

    def _warp_fields(self, images, labels):
        """Warped image fields and (int32) label fields."""
        both = self._warp_coarse(images, labels)
        if both is not None or not images + labels:
            return both or ([], [])
        field = self.dense_field((images + labels)[0].device)
        return ([self._warp_with_dense_field(t, field.to(t.device), 1) for t in images],
                [self._warp_with_dense_field(t, field.to(t.device), 0) for t in labels])

    def _warp_in_place(self, result, img_keys, seg_keys):
        if overrides(self, self._transform, 'elastic_transform', 'dense_field'):
            result.update({k: self.elastic_transform(result[k]) for k in img_keys})
            result.update({k: self.elastic_transform(result[k], order=0).int() for k in seg_keys})
            return
        images, labels = self._warp_fields([result[k] for k in img_keys], [result[k] for k in seg_keys])
        result.update(zip(img_keys, images))
        result.update(zip(seg_keys, labels))

    # image and label fields go together, unless a subclass has its own say in either
    def _together(self):
        return not overrides(self, ElasticField, 'apply_to_img', 'apply_to_seg')

    def apply_to_img(self, result):
        self._warp_in_place(result, result.get('img_fields', ()), result.get('seg_fields', ()) if self._together() else ())

    def apply_to_seg(self, result):
        if not self._together():
            self._warp_in_place(result, (), result.get('seg_fields', ()))
