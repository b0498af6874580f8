"""Half gradients of dense 3D calls, summed brick by brick of the gradient volume: bricks cut by the volume's ends, rois that
overlap, magnify, or lie beyond the kernel's range, gradients that need one word per voxel, two, or flags.  Against the
restatement with a wide accumulator.

The contributions are the restatement's own and their sum is exact, whatever the sizes of the gradients: one rounding to half on
either side, 2^-11 of the value or half a unit of 2^-24 each, and roundings to float far below that."""
import pytest
import torch

import cases
from oracle import port
from test_zz_no_alloc import _call

pytestmark = pytest.mark.gpu

SHAPE = (4, 2, 56, 70, 75)  # 800 bricks, cut on every axis


def make_rois(g, n, zoom, tilt=0.9, shape=SHAPE):
    ext = torch.tensor(shape[:1:-1], dtype=torch.float32)
    b = torch.arange(n).remainder(shape[0]).float().view(-1, 1)
    centre = ext / 2 + (torch.rand(n, 3, generator=g) - 0.5) * ext * 0.3
    size = ext * zoom * (0.85 + 0.3 * torch.rand(n, 3, generator=g))
    return torch.cat([b, centre, size, (torch.rand(n, 3, generator=g) - 0.5) * 2 * tilt], 1).half()


CASES = {
    # rois, zoom, out, order, gradient size, kind
    "one word": dict(n=3, zoom=1.0, out=(48, 70, 66), size=1.0),
    "coarser units": dict(n=3, zoom=1.0, out=(48, 70, 67), size=2.5),
    "two words": dict(n=3, zoom=1.0, out=(48, 66, 71), size=3000.0),
    "peaks": dict(n=3, zoom=1.0, out=(48, 70, 66), size=2e-6, peak=8.0),  # a few large gradients among tiny ones
    "larger peaks": dict(n=3, zoom=1.0, out=(48, 70, 66), size=1e-4, peak=500.0),
    "tiny": dict(n=3, zoom=1.0, out=(48, 66, 70), size=3e-5),
    "turned anyhow": dict(n=3, zoom=1.0, out=(50, 61, 70), size=1.0, tilt=3.1),
    "overlapping": dict(n=8, zoom=0.8, out=(40, 60, 64), size=1.0),
    "large": dict(n=3, zoom=2.4, out=(24, 33, 40), size=1.0),
    "magnified": dict(n=6, zoom=0.8, out=(44, 60, 70), size=1.0, mixed=True),  # a volume with a roi whose steps are below 0.4 voxels
    "nearest": dict(n=3, zoom=1.0, out=(48, 70, 66), size=1.0, order=0),
    "boxes": dict(n=3, zoom=0.9, out=(48, 70, 65), size=1.0, box=True),
    "nearest, two words": dict(n=3, zoom=1.2, out=(48, 70, 66), size=40.0, order=0),
    # several bricks per CTA, the last of them beyond the volume; more rois than threads; no rois in some volumes
    "long columns": dict(n=50, zoom=1.0, out=(36, 33, 38), size=1.0, shape=(50, 4, 40, 36, 36)),
    "longer columns": dict(n=90, zoom=1.0, out=(30, 33, 38), size=12.0, shape=(100, 4, 40, 36, 36)),
    "many rois": dict(n=760, zoom=1.0, out=(15, 17, 18), size=1.0, shape=(800, 1, 16, 16, 16)),
    # about z, where words and rounding errors differ by axis
    "thin": dict(n=4, zoom=1.0, out=(13, 150, 170), size=1.0, shape=(4, 2, 13, 160, 180), flat=True),
    # a step beyond the rules: too few bricks, too thin, an axis of one voxel, rois that touch too few of them
    "739 bricks": dict(n=739, zoom=1.0, out=(15, 17, 18), size=1.0, shape=(739, 1, 16, 16, 16)),
    "740 bricks": dict(n=740, zoom=1.0, out=(15, 17, 18), size=1.0, shape=(740, 1, 16, 16, 16)),
    "eleven planes": dict(n=4, zoom=1.0, out=(11, 150, 170), size=1.0, shape=(4, 2, 11, 160, 180), flat=True),
    "one plane": dict(n=4, zoom=1.0, out=(1, 150, 170), size=1.0, shape=(4, 2, 1, 160, 180), flat=True),
    # turning about z at most, steps on either side of the limit of 0.6 voxels in one call
    "about z, magnified": dict(n=60, zoom=0.57, out=(48, 52, 56), size=1.0, shape=(60, 1, 64, 64, 64), flat=True),
    "small rois": dict(n=4, zoom=0.3, out=(16, 20, 20), size=1.0),
}


@pytest.mark.parametrize("name", CASES)
def test_gradient(name):
    from medvision_b200 import _C
    k = dict(dict(order=1, box=False, tilt=0.9, mixed=False, peak=0.0, shape=SHAPE, flat=False), **CASES[name])
    g = torch.Generator().manual_seed(len(name))
    shape = k["shape"]
    rois = make_rois(g, k["n"], k["zoom"], k["tilt"], shape)
    if k["flat"]:
        rois[:, 7:9] = 0
    if k["mixed"]:
        rois[0, 4:7] *= 0.4
    if k["box"]:
        rois = torch.cat([rois[:, :1], rois[:, 1:4] - rois[:, 4:7] / 2, rois[:, 1:4] + rois[:, 4:7] / 2], 1)
    kind = cases.KIND_BOX if k["box"] else cases.KIND_ROTATED
    out = k["out"]
    grad = (torch.randn((k["n"], shape[1]) + out, generator=g).clamp_(-4, 4) * k["size"]).half()
    if k["peak"]:
        at = torch.randint(0, grad[0].numel(), (40,), generator=g)
        grad.view(k["n"], -1)[:, at] = k["peak"] * torch.randn(40, generator=g).sign().half()
    kw = dict(spatial_scale=1.0, sampling_ratio=1, aligned=not k["box"], order=k["order"], trig=None if k["box"] else port.device_trig(rois))
    # unaligned gradient memory, a result that is added to
    dev = torch.empty(grad.numel() + 1, dtype=torch.half, device="cuda")[1:].view(grad.shape).copy_(grad)
    before = torch.randint(-2, 3, shape, generator=g).half() * k["size"]
    got = before.cuda()
    if k["box"]:
        _C.roi_align_3d_backward(dev, rois.cuda(), got, *out, 1.0, 1, k["order"])
    else:
        _C.roi_align_rotated_3d_backward(dev, rois.cuda(), got, *out, 1.0, 1, True, k["order"])
    want = port.backward(grad, rois, shape, kind, wide_acc=True, **kw).double()
    err = (got.cpu().double() - before.double() - want).abs()
    bound = 2.0 ** -11 * (2 * want.abs() + 2 * (want + before.double()).abs()) + 2.0 ** -24
    assert not bool((err > bound).any()), float((err - bound).max())


def test_infinities_nan_and_bad_batch_index():
    from medvision_b200 import _C
    g = torch.Generator().manual_seed(5)
    rois = make_rois(g, 4, 1.0)
    out = (48, 66, 70)
    grad = torch.randn((4, SHAPE[1]) + out, generator=g).half()
    for r, c, v in ((0, 0, float("inf")), (1, 1, float("-inf")), (2, 0, float("nan")), (2, 1, 60000.0)):
        at = [torch.randint(0, s, (40,), generator=g) for s in out]
        grad[r, c, at[0], at[1], at[2]] = v
    grad[0, 0, 24, 30:33, 35] = torch.tensor([float("inf"), float("-inf"), float("inf")]).half()
    kw = dict(spatial_scale=1.0, sampling_ratio=1, aligned=True, order=1)
    want = port.backward(grad[:3], rois[:3], SHAPE, cases.KIND_ROTATED, wide_acc=True, trig=port.device_trig(rois[:3]), **kw)
    rois[3, 0] = 7
    _C.last_status()
    got = torch.zeros(SHAPE, dtype=torch.half, device="cuda")
    _C.roi_align_rotated_3d_backward(grad.cuda(), rois.cuda(), got, *out, 1.0, 1, True, 1)
    assert _C.last_status() & 1
    got = got.cpu()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    fin = want.isfinite()
    assert bool(((got - want)[fin].abs().double() <= 2.0 ** -10 * want[fin].abs().double() + 2.0 ** -18).all())
    # the sum does not depend on any order
    again = torch.zeros(SHAPE, dtype=torch.half, device="cuda")
    _C.roi_align_rotated_3d_backward(grad.cuda(), rois.cuda(), again, *out, 1.0, 1, True, 1)
    assert torch.equal(again.cpu().view(torch.int16), got.view(torch.int16))
    _C.last_status()


SLOW = {
    # rois per volume, zoom, gradient size, peaks
    "one": (1, 1.0, 1.0, False),
    "loss scale": (1, 1.0, 100.0, False),
    "peaks": (1, 1.0, 10.0, True),
    "magnified": (1, 2.0, 1.0, False),
    "two rois": (2, 1.0, 1.0, False),
    "about z, loss scale": (1, 1.0, 100.0, False),
}


@pytest.mark.parametrize("name", SLOW)
def test_no_call_is_much_slower_than_by_scattering(name):
    """Two volumes of 128^3 against the entry point that always scatters.  2: the bricks' launches, where they find nothing to do or are
    at their least favourable, take up to 1.35 times its time; the least of five, so that a busy host does not count."""
    from medvision_b200 import _lib
    per, zoom, size, peaks = SLOW[name]
    shape = (2, 1, 128, 128, 128)
    g = torch.Generator().manual_seed(3)
    n = 2 * per
    ext = torch.full((n, 3), 128.0)
    angles = (torch.rand(n, 3, generator=g) - 0.5)
    if "about z" in name:
        angles[:, :2] = 0
    b = torch.arange(n).remainder(2).float().view(-1, 1)
    rois = torch.cat([b, ext / 2, ext / zoom, angles], 1).half().cuda()
    grad = torch.randn((n,) + shape[1:], generator=g) * size
    if peaks:
        grad *= torch.where(torch.rand(grad.shape, generator=g) < 1e-4, 1.0, 1e-4)
    grad = grad.half().cuda()
    gin = torch.zeros(shape, dtype=torch.half, device="cuda")
    best = []
    for fn in (_lib.lib.mvr_roi_resample_bwd, _lib.lib.mvr_roi_resample_bwd_noalloc):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200000)  # the launches are queued behind it
            a.record()
            assert _call(fn, grad, rois, gin) == 0
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        best.append(min(times[2:]))
    assert best[0] <= 2 * best[1], best


@pytest.mark.parametrize("order", [1, 0])
@pytest.mark.parametrize("shape,zoom,tilt", [((2, 1, 128, 128, 128), 1.0, 0.0), ((2, 1, 128, 128, 128), 1.1, 1.0), ((4, 1, 90, 100, 110), 1.3, 0.6),
                                             ((8, 1, 13, 180, 200), 1.0, 0.0)])
def test_sums_of_one_sign(shape, zoom, tilt, order):
    """Gradients that are all the same, up to and beyond what one word per voxel holds: the largest sums that the bound of the weights
    allows, against the entry point that scatters into float.  Sums of some tens of contributions differ by 2^-18 there, so one rounding to
    half on either side leaves them one unit apart at most, 2^-10 of the value."""
    from medvision_b200 import _lib
    n = shape[0]
    g = torch.Generator().manual_seed(7)
    ext = torch.tensor(shape[:1:-1], dtype=torch.float32).expand(n, 3)
    angles = (torch.rand(n, 3, generator=g) - 0.5) * tilt
    rois = torch.cat([torch.arange(n).float().view(-1, 1), ext / 2, ext / zoom, angles], 1).half().cuda()
    for value in (2.5, 4.0, 6.0, 8.0, 10.0, 13.0, 16.0, 24.0, -12.0):
        grad = torch.full((n,) + shape[1:], value, dtype=torch.half, device="cuda")
        got = []
        for fn in (_lib.lib.mvr_roi_resample_bwd, _lib.lib.mvr_roi_resample_bwd_noalloc):
            gin = torch.zeros(shape, dtype=torch.half, device="cuda")
            assert fn(grad.data_ptr(), rois.data_ptr(), gin.data_ptr(), _lib.MVR_F16, 3, _lib.MVR_ROI_ROTATED, *shape, n, 10, *shape[2:], 1.0, 1, 1,
                      order, None, torch.cuda.current_stream().cuda_stream) == 0
            got.append(gin.double())
        assert bool(((got[0] - got[1]).abs() <= 2.0 ** -10 * got[1].abs() + 2.0 ** -24).all()), value
