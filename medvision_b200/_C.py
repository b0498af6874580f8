"""The resampling functions of the reference's compiled extension, on torch tensors: the ten
roi / affine functions and ``deform_2d`` / ``deform_3d`` in the configuration ``apply_offset_*`` uses.

Same names, argument order and error behaviour as ``medvision._C``
(medvision/csrc/vision.cpp:34-48,74-75 and the dispatch headers medvision/csrc/roi_align_*.h,
affine_*.h): every function returns ``None`` and writes into a caller-allocated tensor;
a non-CUDA input raises ``RuntimeError("... is not implemented on CPU")``; a wrong roi width
raises ``RuntimeError("wrong roi size! size_rois should be K")``.

Differences from the reference, all deliberate: the launch goes to torch's CURRENT stream of
the input's device under a device guard (the reference launches on the legacy default stream of
whatever device is current); flat offsets are 64-bit; an empty roi list is a no-op (the reference
fails with a zero-block launch); a roi whose batch index lies outside the batch yields zeros and
sets a status bit (see :func:`last_status`) instead of reading out of bounds.

Checks, allocation and launches are native (csrc/mvr_torch.cpp, compiled into ``_native.so``): a call costs 2-3 us of
CPU time with its launch, where the same through ctypes took 8 us.
"""
import torch

from . import _lib      # raises when libmvr.so is missing
from . import _native   # the host path; links libmvr.so


def last_status(device=None, clear=True):
    """Status bits OR-ed by the kernels launched on ``device`` so far (synchronises)."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    w = _native.status_word(device.index if device.index is not None else torch.cuda.current_device())
    v = int(w.item())
    if clear:
        w.zero_()
    return v


def cached_memory_bytes(device=None):
    """Bytes held by the library's memory pool on ``device`` (the float accumulator volumes of the dense 3D half
    backward come from it; it keeps up to 1 GiB between calls)."""
    index = torch.cuda.current_device() if device is None else torch.device(device).index
    with torch.cuda.device(index):
        return int(_lib.lib.mvr_cached_memory_bytes())


def release_cached_memory(device=None):
    """Give the unused part of that pool, and the buffers through which the transforms' rois are uploaded, back to the
    driver."""
    index = torch.cuda.current_device() if device is None else torch.device(device).index
    with torch.cuda.device(index):
        rc = _lib.lib.mvr_release_cached_memory()
        _native.release_staging(index)
    if rc != 0:
        raise RuntimeError(_lib.strerror(rc))


_call = _native.roi_call
_BOX, _ROTATED = _lib.MVR_ROI_BOX, _lib.MVR_ROI_ROTATED


def roi_align_2d_forward(input, rois, output, aligned_height, aligned_width, spatial_scale, sampling_ratio, order):
    _call(_BOX, 2, True, False, input, rois, output, (aligned_height, aligned_width),
          spatial_scale, sampling_ratio, False, order)


def roi_align_2d_backward(top_grad, rois, bottom_grad, aligned_height, aligned_width, spatial_scale, sampling_ratio,
                          order):
    _call(_BOX, 2, False, False, top_grad, rois, bottom_grad, (aligned_height, aligned_width),
          spatial_scale, sampling_ratio, False, order)


def roi_align_3d_forward(input, rois, output, aligned_depth, aligned_height, aligned_width, spatial_scale,
                         sampling_ratio, order):
    _call(_BOX, 3, True, False, input, rois, output, (aligned_depth, aligned_height, aligned_width),
          spatial_scale, sampling_ratio, False, order)


def roi_align_3d_backward(top_grad, rois, bottom_grad, aligned_depth, aligned_height, aligned_width, spatial_scale,
                          sampling_ratio, order):
    _call(_BOX, 3, False, False, top_grad, rois, bottom_grad, (aligned_depth, aligned_height, aligned_width),
          spatial_scale, sampling_ratio, False, order)


def roi_align_rotated_2d_forward(input, rois, output, aligned_height, aligned_width, spatial_scale, sampling_ratio,
                                 aligned, order):
    _call(_ROTATED, 2, True, False, input, rois, output, (aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


def roi_align_rotated_2d_backward(top_grad, rois, bottom_grad, aligned_height, aligned_width, spatial_scale,
                                  sampling_ratio, aligned, order):
    _call(_ROTATED, 2, False, False, top_grad, rois, bottom_grad, (aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


def roi_align_rotated_3d_forward(input, rois, output, aligned_depth, aligned_height, aligned_width, spatial_scale,
                                 sampling_ratio, aligned, order):
    _call(_ROTATED, 3, True, False, input, rois, output, (aligned_depth, aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


def roi_align_rotated_3d_backward(top_grad, rois, bottom_grad, aligned_depth, aligned_height, aligned_width,
                                  spatial_scale, sampling_ratio, aligned, order):
    _call(_ROTATED, 3, False, False, top_grad, rois, bottom_grad, (aligned_depth, aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


def affine_2d(input, rois, output, aligned_height, aligned_width, spatial_scale, sampling_ratio, aligned, order):
    _call(_ROTATED, 2, True, True, input, rois, output, (aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


def affine_3d(input, rois, output, aligned_depth, aligned_height, aligned_width, spatial_scale, sampling_ratio,
              aligned, order):
    _call(_ROTATED, 3, True, True, input, rois, output, (aligned_depth, aligned_height, aligned_width),
          spatial_scale, sampling_ratio, aligned, order)


_LABEL_DTYPES = {torch.uint8: 0, torch.int16: 1, torch.int32: 2, torch.int64: 3}


def affine_label(input, rois, output, out_sizes, spatial_scale, aligned):
    """Nearest resampling of an integer label tensor into an int32 ``output``: the result of the
    reference's ``affine_*(input.float(), rois, ..., order=0).int()`` without the float copies.
    ``rois`` is float32.  Not a function of the reference's extension.  Returns False when the
    library has no label kernel for the shape (the caller then takes the cast path)."""
    return _native.label_call(input, rois, output, tuple(out_sizes), spatial_scale, aligned)


def affine_fields_3d(image, image_rois, image_out, labels, label_rois, label_out, out_sizes, spatial_scale, aligned,
                     order):
    """An image field and its label field of one augmentation call: ``affine_3d(image, image_rois, ...,
    sampling_ratio 1)`` into ``image_out`` and :func:`affine_label` of ``labels`` (float32 ``label_rois``, the same
    rois) into the int32 ``label_out``, with the label's work riding along with the image's launches where the
    shapes allow.  Not a function of the reference's extension."""
    _native.fields_call(image, image_rois, image_out, labels, label_rois, label_out, tuple(out_sizes), spatial_scale, aligned,
                        order)


def apply_offset(input, offset, order):
    """Displacement-field warp: ``out[b, c, p] = interp(input[b, c], p + offset[b, :, p])``.  Not a
    function of the reference's extension: it is what ``deform_2d`` / ``deform_3d`` compute in the
    configuration ``apply_offset_2d/3d`` call them with.  A float32 field with a half image is
    rounded to half as it is read (the reference casts it in a pass of its own)."""
    return _native.apply_offset(input, offset, order)


def _deform(name, ndim, input, weight, bias, offset, geometry, group, deformable_groups, order):
    """The reference's ``deform_2d`` / ``deform_3d`` (medvision/csrc/vision.cpp:76-77) for the one
    configuration its Python layer uses (medvision/ops/cuda_fun_tools.py:94-167): 1x1(x1) kernel,
    stride 1, no padding, dilation 1, one group, one deformable group, identity weight and zero
    bias -- i.e. a displacement-field warp.  ``weight`` and ``bias`` are accepted for signature
    compatibility; anything but that configuration is refused."""
    kernel, stride, padding, dilation = geometry
    if not (all(k == 1 for k in kernel) and all(v == 1 for v in stride) and all(v == 0 for v in padding)
            and all(v == 1 for v in dilation) and group == 1 and deformable_groups == 1):
        raise NotImplementedError(f"{name}: only the 1x1 identity configuration of apply_offset_* is provided")
    if not input.is_cuda:
        raise RuntimeError("Not implemented on the CPU")
    if input.dim() != ndim + 2:
        raise RuntimeError(f"{name}: expected a {ndim + 2}-D input")
    if tuple(weight.shape) != (input.size(1), input.size(1)) + (1,) * ndim:
        raise NotImplementedError(f"{name}: the weight must be the channel identity")
    if offset.dtype != input.dtype:
        # the reference reinterprets with tensor.data<scalar_t>(), which throws on a mismatch
        raise RuntimeError(f"expected scalar type {input.dtype} but found {offset.dtype}")
    return apply_offset(input, offset, order)


def deform_2d(input, weight, bias, offset, kernel_h, kernel_w, stride_h, stride_w, pad_h, pad_w, dilation_h,
              dilation_w, group, deformable_groups, im2col_step, order):
    return _deform("deform_2d", 2, input, weight, bias, offset,
                   ((kernel_h, kernel_w), (stride_h, stride_w), (pad_h, pad_w), (dilation_h, dilation_w)),
                   group, deformable_groups, order)


def deform_3d(input, weight, bias, offset, kernel_d, kernel_h, kernel_w, stride_d, stride_h, stride_w, pad_d, pad_h,
              pad_w, dilation_d, dilation_h, dilation_w, group, deformable_groups, im2col_step, order):
    return _deform("deform_3d", 3, input, weight, bias, offset,
                   ((kernel_d, kernel_h, kernel_w), (stride_d, stride_h, stride_w), (pad_d, pad_h, pad_w),
                    (dilation_d, dilation_h, dilation_w)), group, deformable_groups, order)
