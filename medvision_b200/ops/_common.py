"""What the roi operations share: the parsing of an output size, and the base of their autograd Functions."""
from torch.autograd import Function


def parse_output_size(output_size, ndim, name="output_size"):
    """int -> the same size on every axis; tuple of ``ndim`` ints -> as given.  Anything else
    (a list included) is a TypeError, as in medvision/ops/roi_align_nd.py:14-26."""
    if isinstance(output_size, int):
        return (output_size,) * ndim
    if isinstance(output_size, tuple):
        assert len(output_size) == ndim
        for v in output_size:
            assert isinstance(v, int)
        return output_size
    raise TypeError(f'"{name}" must be an integer or tuple of integers')


class RoiFunction(Function):
    """Base of the autograd Functions of medvision/ops/roi_align_nd.py:13-133 and roi_align_rotated_nd.py:13-161.

    ``apply`` of the operations' own classes is the native call ``call`` with its native autograd node (csrc/mvr_torch.cpp).  A
    class derived from one of them, with a forward or backward of its own, goes through torch's Function as usual, on the extension
    functions ``kernels``."""
    ndim, call, kernels = 0, None, ()

    @classmethod
    def apply(cls, *args, **kwargs):
        if "call" in cls.__dict__:
            return cls.call(*args, **kwargs)
        return super().apply(*args, **kwargs)

    @classmethod
    def _forward(cls, ctx, features, rois, output_size, spatial_scale, sampling_ratio, *options):
        out = parse_output_size(output_size, cls.ndim)
        assert features.dim() == cls.ndim + 2
        ctx.geometry = spatial_scale, sampling_ratio, *options
        ctx.feature_size = features.size()
        ctx.save_for_backward(rois)
        output = features.new_empty((rois.size(0), features.size(1)) + tuple(out))
        cls.kernels[0](features, rois, output, *out, *ctx.geometry)
        return output

    @classmethod
    def _backward(cls, ctx, grad_output):
        rois, = ctx.saved_tensors
        grad_input = None
        if ctx.needs_input_grad[0]:
            grad_input = rois.new_zeros(ctx.feature_size)  # the rois' dtype, as in the reference
            cls.kernels[1](grad_output.contiguous(), rois, grad_input, *grad_output.shape[2:], *ctx.geometry)
        return (grad_input,) + (None,) * (len(ctx.geometry) + 2)
