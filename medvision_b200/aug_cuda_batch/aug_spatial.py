"""Batched geometric augmentations built on the resampling op.

Same classes, constructor arguments, parameter draws and roi formulas as the resampling
transforms of medvision/aug_cuda_batch/aug_spatial.py (Resize :69-194, RandomAffine / Scale /
Shift / Rotate :355-597, Crop*WithAffine :600-957).  What differs:
  * the rois of a call are built once (float32 on the host, in the reference's operation order,
    so the values are the same) and shared by the image and the label fields;
  * ``times`` crops per image address the SAME image through the roi's batch index instead of
    concatenating ``times`` copies of the batch;
  * label fields go through the nearest-neighbour path of the same kernel.
"""
import random
from typing import Union

import numpy as np
import torch

from .base import BatchCudaAugBase, global_bit_generator
from .elastic_field import ElasticField
from .. import _C


def _resample_fields(result, dim, rois, out_size, sampling_ratio, order):
    """All image and label fields of ``result`` through the rois of this call (CPU float32), in one native call: the rois
    go to the device once (one asynchronous copy, float32 and float16 at once); in 3D an image field and a label field are
    resampled by one fused launch pair whose label work rides along with the image's."""
    assert not result.get('det_fields'), 'detection boxes are not handled by the resampling transforms'
    img_keys, seg_keys = result.get('img_fields', ()), result.get('seg_fields', ())
    images, labels = _C._native.resample_fields(dim, [result[k] for k in img_keys], [result[k] for k in seg_keys], rois,
                                                tuple(int(v) for v in out_size), sampling_ratio, order)
    result.update(zip(img_keys, images))
    result.update(zip(seg_keys, labels))


def _affine_rois(t, n_images, image_shape, start=None, end=None):
    """[image, center - shape * shifts / scales, shape / scales, angles] of every sample of the transform ``t`` in float32
    (rotation about z in 3D): over the whole image, or over the patches start..end (xyz)."""
    p = [np.ascontiguousarray(t.params[k], dtype=np.float64) for k in ("scales", "shifts", "rotate")]
    if start is not None:
        start, end = (np.ascontiguousarray(v, dtype=np.int64) for v in (start, end))
    return _C._native.affine_rois(len(p[0]), t.dim, n_images, *p, None if image_shape is None else tuple(image_shape), start, end)


def _whole_image(image_shape):
    """Centre and extent (float32, xyz) of a (d,) h, w shape."""
    shape = np.array(image_shape[::-1], dtype=np.float32)
    return shape / 2, shape


class BatchCudaResize(BatchCudaAugBase):
    def __init__(self, spacing=None, scale=None, factor=None, order=1):
        super().__init__()
        self.always = True
        self.spacing = spacing
        self.scale = scale
        self.factor = factor
        self.order = order
        assert sum([spacing is not None, scale is not None, factor is not None]) == 1

    def __repr__(self):
        return self.__class__.__name__ + '(spacing={}, scale={}, factor={})'.format(self.spacing, self.scale, self.factor)

    @property
    def canBackward(self):
        return True

    def _forward_params(self, result):
        self._init_params(result)
        if self.spacing is not None:
            assert len(self.spacing) == self.dim, f"not match with a {result['img_dim']}D image"
            img_spacing = np.array(result['img_spacing'])
            new_spacing = np.array(self.spacing)
            new_spacing = np.where(new_spacing == -1, img_spacing, new_spacing)
            scale_factor = tuple(img_spacing / new_spacing)
        elif self.scale is not None:
            assert len(self.scale) == self.dim, f"not match with a {result['img_dim']}D image"
            new_shape = np.array(self.scale)
            new_shape = np.where(new_shape == -1, self.image_shape, new_shape)
            scale_factor = tuple(new_shape / self.image_shape)
        else:
            assert len(self.factor) == self.dim, f"not match with a {result['img_dim']}D image"
            scale_factor = tuple(self.factor)
        self.params = scale_factor
        result[self.key_name] = self.params

    def _backward_params(self, result):
        self._init_params(result)
        params = result.pop(self.key_name, None)
        if params:
            self.params = tuple(1 / np.array(params))

    def _rois(self):
        rois = np.zeros((self.batch, 2 * self.dim + (2 if self.dim == 2 else 4)), dtype=np.float32)
        rois[:, 0] = np.arange(self.batch)
        rois[:, 1:1 + self.dim], rois[:, 1 + self.dim:1 + 2 * self.dim] = _whole_image(self.image_shape)
        return torch.from_numpy(rois)

    def apply_to_img(self, result):
        # the whole image is one roi; image and label fields share it
        if all(i == 1.0 for i in self.params):
            return
        out_size = tuple(int(i * p) for i, p in zip(self.image_shape, self.params))
        _resample_fields(result, self.dim, self._rois(), out_size, 1, self.order)

    def apply_to_seg(self, result):
        pass  # done together with the images


class BatchCudaRandomAffine(BatchCudaAugBase):
    def __init__(self, p, scale: Union[float, list, tuple], shift: Union[float, list, tuple],
                 rotate: Union[float, list, tuple], sampling_ratio=1, order=1):
        super().__init__()
        self.p = p
        self.scale = scale
        self.shift = shift
        self.rotate = rotate  # degrees, in the xy plane
        self.sampling_ratio = sampling_ratio
        self.order = order

    def __repr__(self):
        return self.__class__.__name__ + '(dim={}, scale={}, shift={}, rotate={})'.format(
            self.dim, self.scale, self.shift, self.rotate)

    def _forward_params(self, result):
        self._init_params(result)
        scales, shifts, rotate = self._draw_affine(self.batch)
        self.params = {"scales": scales, "shifts": shifts, "rotate": rotate}
        result[self.key_name] = self.params

    def _backward_params(self, result: dict):
        self._init_params(result)
        params = result.get(self.key_name, None)
        if params:
            self.params = {"scales": 1 / params["scales"], "shifts": -params["shifts"], "rotate": -params["rotate"]}

    def _rois(self):
        return _affine_rois(self, self.batch, self.image_shape)

    def apply_to_img(self, result: dict):
        _resample_fields(result, self.dim, self._rois(), self.image_shape, self.sampling_ratio, self.order)

    def apply_to_seg(self, result: dict):
        pass  # done together with the images


class BatchCudaRandomScale(BatchCudaRandomAffine):
    def __init__(self, p, scale: Union[float, list, tuple], sampling_ratio=1):
        super().__init__(p, scale=scale, shift=0, rotate=0, sampling_ratio=sampling_ratio)


class BatchCudaRandomShift(BatchCudaRandomAffine):
    def __init__(self, p, shift: Union[float, list, tuple], sampling_ratio=1):
        super().__init__(p, scale=0, shift=shift, rotate=0, sampling_ratio=sampling_ratio)


class BatchCudaRandomRotate(BatchCudaRandomAffine):
    def __init__(self, p, rotate: Union[float, list, tuple], sampling_ratio=1):
        super().__init__(p, scale=0, shift=0, rotate=rotate, sampling_ratio=sampling_ratio)


class BatchCudaRandomElasticDeformation(ElasticField, BatchCudaAugBase):
    """Random smooth warp, as medvision/aug_cuda_batch/aug_spatial.py:204-313: a coarse grid of
    ``num_control_points`` random displacements per sample (at most ``max_displacement`` half grid
    cells, the two outermost control points of every axis locked to zero), interpolated to every voxel
    (order ``order``, Catmull-Rom by default) and applied -- linear for images, nearest for labels.
    ``dense_field`` / ``tmp_params`` is the (B, dim, *image_shape) field itself, made when it is asked
    for; ``backward`` negates the coarse field."""

    def __init__(self, p, num_control_points=8, max_displacement: float = 0.8, order=3):
        super().__init__()
        self.p = p
        self.num_control_points = num_control_points  # d, h, w order
        self.max_displacement = max_displacement
        self.INTER_ORDER = order
        self.num_locked_borders = 2
        assert max_displacement <= 1.0

    def __repr__(self):
        return self.__class__.__name__ + "(p={}, num_control_points={}, max_displacement={})".format(
            self.p, self.num_control_points, self.max_displacement)

    @property
    def canBackward(self):
        return True

    @property
    def _field_order(self):
        return self.INTER_ORDER

    def _forward_params(self, result):
        self.tmp_params = None
        self._init_params(result)
        self.params = self._draw_coarse(self.batch)
        result[self.key_name] = self.params

    def _backward_params(self, result):
        self.tmp_params = None
        self._init_params(result)
        params = result.pop(self.key_name, None)
        if params is not None:
            self.params = -params

    def dense_field(self, device):
        """(B, dim, *image_shape) float32 displacement field on ``device``."""
        if self._dense is None:
            self._dense = self._blow_up(device)
        return self._dense

    def elastic_transform(self, image: torch.Tensor, order=1):
        """One field (B, C, *image_shape) by the dense field."""
        return self._warp_with_dense_field(image, self.dense_field(image.device), order)

    def apply_to_det(self, result):
        for key in result.get('det_fields', []):
            raise NotImplementedError


BatchCudaRandomElasticDeformation._transform = BatchCudaRandomElasticDeformation


class BatchCudaCropRandomWithAffine(BatchCudaAugBase):
    def __init__(self, patch_size, scale: Union[float, list, tuple], shift: Union[float, list, tuple],
                 rotate: Union[float, list, tuple], sampling_ratio=1, order=1, times=1):
        super().__init__()
        self.always = True
        self.dim = len(patch_size)
        self.patch_size = patch_size
        self.scale = scale
        self.shift = shift
        self.rotate = rotate
        self.sampling_ratio = sampling_ratio
        self.order = order
        self.times = times

    def __repr__(self):
        return self.__class__.__name__ + "(patch_size={})".format(self.patch_size)

    @property
    def repeats(self):
        return self.times

    def _init_params(self, result):
        super()._init_params(result)
        self.n_images = self.batch
        self.batch = self.n_images * self.times  # one parameter set per produced patch

    def _forward_params(self, result):
        self._init_params(result)
        assert self.dim == len(self.patch_size)
        assert all(self.image_shape[i] >= self.patch_size[i] for i in range(self.dim)), self.image_shape
        batch_start, batch_end = self._forward_crop_params(result)
        batch_scales, batch_shifts, batch_rotate = self._forward_affine_params(result)
        self.params = {"start": batch_start, "end": batch_end,  # xyz
                       "scales": batch_scales, "shifts": batch_shifts, "rotate": batch_rotate}
        result[self.key_name] = self.params

    def _forward_affine_params(self, result: dict):
        return self._draw_affine(self.batch)

    def _random_start(self):
        return tuple(map(lambda a, da: np.random.randint(0, a - da + 1), self.image_shape, self.patch_size))

    def _start_near(self, obj):
        """a patch start such that the patch covers the object ``obj`` (slices, dhw) with a border"""
        lo = tuple(min(max(obj[d].stop + self.border - self.patch_size[d], 0), self.image_shape[d] - self.patch_size[d])
                   for d in range(len(obj)))
        hi = tuple(min(max(obj[d].start - self.border, 0), self.image_shape[d] - self.patch_size[d])
                   for d in range(len(obj)))
        return tuple(map(lambda a, da: np.random.randint(min(a, da), max(a, da) + 1), lo, hi))

    def _collect(self, starts):
        batch_start = [s[::-1] for s in starts]
        batch_end = [tuple(a + b for a, b in zip(s, self.patch_size))[::-1] for s in starts]
        return np.array(batch_start), np.array(batch_end)

    def _forward_crop_params(self, result: dict):
        if getattr(self._random_start, '__func__', None) is not BatchCudaCropRandomWithAffine._random_start:
            return self._collect([self._random_start() for _ in range(self.batch)])
        # one draw per patch and axis (d, h, w), as _random_start() makes them
        start = np.empty((self.batch, self.dim), dtype=np.int64)
        end = np.empty_like(start)
        generator = global_bit_generator()
        with generator.lock:
            _C._native.draw_starts(generator.capsule, self.batch, tuple(self.image_shape), tuple(self.patch_size), start, end)
        return start, end

    def _rois(self):
        # patch r*B + b is cut from image b
        return _affine_rois(self, self.n_images, None, self.params["start"], self.params["end"])

    def apply_to_img(self, result: dict):
        _resample_fields(result, self.dim, self._rois(), self.patch_size, self.sampling_ratio, self.order)

    def apply_to_seg(self, result: dict):
        pass  # done together with the images


class BatchCudaCropCenterWithAffine(BatchCudaCropRandomWithAffine):
    def _forward_crop_params(self, result: dict):
        start = tuple(map(lambda a, da: a // 2 - da // 2, self.image_shape, self.patch_size))
        return self._collect([start for _ in range(self.batch)])


class BatchCudaCropForegroundWithAffine(BatchCudaCropRandomWithAffine):
    def __init__(self, border=12, **kwargs):
        super().__init__(**kwargs)
        self.border = border

    def _forward_crop_params(self, result: dict):
        import scipy.ndimage as ndi
        assert 'gt_seg' in result.keys() or 'pseudo_mask' in result.keys()
        mask = result['gt_seg'] if 'gt_seg' in result.keys() else result['pseudo_mask']
        starts = []
        for i in range(self.batch):
            foreground = mask[i % self.n_images, 0]
            if torch.is_tensor(foreground):
                foreground = foreground.cpu().numpy()
            objs = ndi.find_objects(ndi.label(foreground)[0])
            starts.append(self._start_near(random.choice(objs)) if len(objs) else self._random_start())
        return self._collect(starts)


class BatchCudaCropDetWithAffine(BatchCudaCropRandomWithAffine):
    """patches around the ground-truth boxes, one box after the other over the repeats"""

    def __init__(self, border=12, **kwargs):
        super().__init__(**kwargs)
        self.border = border
        self.current_repeat_idx = 0

    def _box(self, result, k):
        obj = result['gt_det'][k]
        return [slice(int(obj[self.dim - i - 1]), int(obj[2 * self.dim - i - 1])) for i in range(self.dim)]

    def _forward_crop_params(self, result: dict):
        assert 'gt_det' in result.keys(), "it only used for detection tasks"
        starts = []
        for _ in range(self.batch):
            k = min(self.current_repeat_idx % self.repeats, len(result['gt_det']) - 1)
            self.current_repeat_idx += 1
            starts.append(self._start_near(self._box(result, k)))
        return self._collect(starts)


class BatchCudaCropFirstDetWithAffine(BatchCudaCropDetWithAffine):
    def _forward_crop_params(self, result: dict):
        assert 'gt_det' in result.keys(), "it only used for detection tasks"
        return self._collect([self._start_near(self._box(result, 0)) for _ in range(self.batch)])
