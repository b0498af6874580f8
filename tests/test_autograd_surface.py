"""The roi operations as autograd Functions: class relations, subclasses with code of their own, saved-tensor hooks, and the
transforms of torch that they refuse."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from medvision_b200.ops import roi_align_nd, roi_align_rotated_nd

CLASSES = [roi_align_nd.RoIAlign2DFunction, roi_align_nd.RoIAlign3DFunction, roi_align_rotated_nd.RoIAlignRotated2DFunction,
           roi_align_rotated_nd.RoIAlignRotated3DFunction]


def _inputs(cls, device="cpu"):
    nd = cls.ndim
    g = torch.Generator().manual_seed(nd)
    x = torch.rand((1, 2) + (12,) * nd, generator=g)
    centre, size = torch.full((3, nd), 6.0), torch.rand(3, nd, generator=g) * 6 + 2
    if "Rotated" in cls.__name__:
        rois = torch.cat([torch.zeros(3, 1), centre, size, torch.rand(3, 1 if nd == 2 else 3, generator=g)], 1)
    else:
        rois = torch.cat([torch.zeros(3, 1), centre - size / 2, centre + size / 2], 1)
    return x.to(device), rois.to(device), (3,) * nd, 1.0, 2


@pytest.mark.parametrize("cls", CLASSES)
def test_they_are_functions(cls):
    assert issubclass(cls, torch.autograd.Function)
    with pytest.raises(RuntimeError, match="not implemented on CPU"):
        cls.apply(*_inputs(cls))

    class Derived(cls):
        @staticmethod
        def forward(ctx, *args):
            ctx.seen = True
            return cls.forward(ctx, *args)

    with pytest.raises(RuntimeError, match="not implemented on CPU"):
        Derived.apply(*_inputs(cls))
    with pytest.raises(TypeError, match="must be an integer or tuple of integers"):
        Derived.apply(*_inputs(cls)[:2], [3] * cls.ndim, 1.0)


@pytest.mark.gpu
@pytest.mark.parametrize("cls", CLASSES)
def test_subclasses_and_hooks(cls):
    x, *args = _inputs(cls, "cuda")
    x.requires_grad_()
    want = cls.apply(x, *args)
    grad = torch.rand_like(want)
    want_grad, = torch.autograd.grad(want, x, grad)

    class Halved(cls):
        @staticmethod
        def forward(ctx, *args):
            return cls.forward(ctx, *args) / 2

        @staticmethod
        def backward(ctx, grad_output):
            return cls.backward(ctx, grad_output / 2)

    got = Halved.apply(x, *args)
    assert torch.equal(got, want / 2)
    torch.testing.assert_close(torch.autograd.grad(got, x, grad)[0], want_grad / 2, rtol=1e-5, atol=1e-7)
    packed = []

    def pack(t):
        packed.append(t)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        out = cls.apply(x, *args)
    torch.testing.assert_close(torch.autograd.grad(out, x, grad)[0], want_grad, rtol=1e-5, atol=1e-7)
    assert len(packed) == 1 and packed[0].shape == args[0].shape
    args[0] = args[0].clone()
    out = cls.apply(x, *args)
    args[0].add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, x, grad)


@pytest.mark.gpu
@pytest.mark.parametrize("cls", CLASSES)
def test_transforms_without_a_rule_are_refused(cls):
    x, *args = _inputs(cls, "cuda")
    with fwAD.dual_level():
        with pytest.raises(RuntimeError):
            cls.apply(fwAD.make_dual(x, torch.ones_like(x)), *args)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: cls.apply(t, *args).sum())(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: cls.apply(t, *args))(x[None])
