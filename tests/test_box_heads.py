"""The box-head kernels (csrc/mvr_head.cuh) at the sizes where their dispatch and their tables change: adaptive and three-sample
grids, boxes from below one voxel to beyond the tables, boxes over the border and outside, channel groups, row widths, odd
maps, unaligned gradient tensors.  Forward bit for bit, backward against the wide-accumulator restatement."""
import pytest
import torch

import cases
from oracle import port
from util import REF_FM, assert_close, assert_half_sums, n_mismatch

pytestmark = pytest.mark.gpu

CASES = [
    # spatial,        channels, rois, output,    sampling, order, dtype, half additions per roi and voxel
    ((37, 41),        5, 12, (7, 7),    0, 1, torch.float32, 0),
    ((600, 530),      1, 9,  (7, 5),    0, 1, torch.float32, 0),   # boxes wider than the tables of positions and of taps
    ((64, 97),        2, 40, (14, 14),  3, 1, torch.float32, 0),   # groups of two
    ((50, 63),        3, 9,  (3, 33),   0, 1, torch.float32, 0),   # rows wider than a warp
    ((37, 41),        4, 12, (7, 7),    0, 0, torch.float32, 0),   # nearest
    ((37, 41),        5, 40, (7, 7),    0, 1, torch.float32, 0),   # enough outputs for a row per warp
    ((37, 41),        4, 40, (7, 7),    0, 0, torch.float32, 0),
    ((600, 530),      2, 90, (7, 7),    0, 1, torch.float32, 0),
    ((70, 2100),      4, 40, (7, 7),    0, 1, torch.float32, 0),   # samples beyond the forward's tables
    ((33, 27),        3, 60, (7, 7),    0, 1, torch.float16, 1),
    ((64, 97),        6, 90, (14, 14),  2, 1, torch.float16, 4),
    ((19, 23, 29),    7, 80, (7, 6, 5), 3, 1, torch.float32, 0),
    ((19, 23, 29),    9, 60, (7, 6, 5), 0, 1, torch.float32, 0),   # enough outputs for the 3D tables
    ((12, 40, 170),   2, 30, (5, 5, 5), 0, 1, torch.float16, 64),   # an axis beyond the tables of positions
    ((19, 23, 29),    3, 40, (7, 7, 7), 2, 0, torch.float16, 8),
    ((640, 700),      2, 30, (5, 4),    0, 1, torch.float16, 16),   # maps beyond the tables: several blocks per box, some idle
    ((200, 336),      5, 30, (7, 7),    2, 1, torch.float16, 4),   # samples far apart beside samples close together
    ((200, 336),      4, 60, (14, 14),  3, 1, torch.float32, 0),
    ((40, 60, 70),    12, 50, (7, 7, 7), 2, 1, torch.float32, 0),  # the same in 3D
    ((64, 80, 96),    2, 20, (4, 5, 6), 2, 0, torch.float16, 8),
]


def _rois(spatial, R, g):
    nd = len(spatial)
    ext = torch.tensor(spatial[::-1], dtype=torch.float32)
    b = torch.randint(0, 2, (R, 1), generator=g).float()
    c = torch.rand(R, nd, generator=g) * ext * 1.1 - 0.05 * ext
    s = torch.rand(R, nd, generator=g) * ext * 0.5 + 0.5
    s[0] = 0.2                        # below one voxel
    s[1] = ext * 2.5                  # the whole map and beyond
    c[1] = ext / 2
    c[2] = ext * 3                    # outside
    c[3], s[3] = ext - 0.5, 3.0       # the last voxels
    c[4], s[4] = torch.zeros(nd), 4.0
    s[5], c[5] = 2.0, ext / 3         # far fewer voxels than bins
    return torch.cat([b, c - s / 2, c + s / 2], 1)


@pytest.mark.parametrize("spatial,C,R,out,sr,order,dtype,adds", CASES,
                         ids=["%s-%s-s%d-o%d-%s" % ("x".join(map(str, c[0])), "x".join(map(str, c[3])), c[4], c[5], str(c[6])[6:]) for c in CASES])
def test_box_heads_match_the_restatement(spatial, C, R, out, sr, order, dtype, adds):
    from medvision_b200 import _C
    nd = len(spatial)
    g = torch.Generator().manual_seed(sum(spatial) + R)
    feat = (torch.rand((2, C) + spatial, generator=g) * 2 - 0.5).to(dtype)
    rois = _rois(spatial, R, g).to(dtype)
    bad = rois.clone()
    bad[6, 0] = 5                     # batch index outside the batch
    fwd = _C.roi_align_2d_forward if nd == 2 else _C.roi_align_3d_forward
    bwd = _C.roi_align_2d_backward if nd == 2 else _C.roi_align_3d_backward
    kw = dict(spatial_scale=1.0, sampling_ratio=sr, aligned=True, order=order, fma_mode=REF_FM if dtype == torch.float32 else 0)
    keep = [i for i in range(R) if i != 6]
    got = torch.full((R, C) + out, float("nan"), dtype=dtype, device="cuda")
    fwd(feat.cuda(), bad.cuda(), got, *out, 1.0, sr, order)
    assert not bool(got[6].any())
    assert n_mismatch(got[keep], port.forward(feat, rois[keep], out, cases.KIND_BOX, **kw)) == 0
    grad = torch.randn((R, C) + out, generator=g).to(dtype)
    want = port.backward(grad[keep], rois[keep], feat.shape, cases.KIND_BOX, wide_acc=True, **kw)
    n = feat.numel()
    for offset in (0, 3):             # a gradient tensor at an unaligned place inside a buffer
        buf = torch.full((n + 32,), -0.0, dtype=dtype, device="cuda")
        gin = buf[16 + offset:16 + offset + n].view(feat.shape)
        gin.zero_()
        bwd(grad.cuda(), bad.cuda(), gin, *out, 1.0, sr, order)
        if dtype == torch.float32:
            assert_close(gin, want, 1e-5, "gradient")
        else:
            assert_half_sums(gin, want, grad[keep], rois[keep], cases.KIND_BOX, adds, **kw)
        around = torch.cat([buf[:16 + offset], buf[16 + offset + n:]])
        assert bool((torch.signbit(around) & (around == 0)).all()), "something was added outside the gradient tensor"
    _C.last_status()


def test_half_gradient_divides_by_the_count_in_half():
    """A bin of more than 255 pixels a side has more samples than half can count: the reference divides by infinity."""
    from medvision_b200 import _C
    rois = torch.tensor([[0, 10, 12, 310, 312], [0, 10, 12, 110, 132]]).half()
    grad = torch.randn(2, 3, 1, 1, generator=torch.Generator().manual_seed(2)).half()
    want = port.backward(grad, rois, (1, 3, 330, 340), cases.KIND_BOX, spatial_scale=1.0, sampling_ratio=0, aligned=True, order=1,
                         wide_acc=True, fma_mode=0)
    assert bool(want[0, :, 50, 50].any()) and not bool(want[0, :, 200, 200].any())
    gin = torch.zeros(want.shape, dtype=torch.half, device="cuda")
    _C.roi_align_2d_backward(grad.cuda(), rois.cuda(), gin, 1, 1, 1.0, 0, 1)
    assert_close(gin, want, 2e-3, "gradient")


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("spatial,C,R,out,sr,rotated", [
    ((64, 97), 3, 90, (14, 14), 2, False),
    ((64, 97), 2, 60, (7, 7), 0, False),
    ((600, 530), 1, 40, (7, 7), 0, False),
    ((19, 23, 29), 7, 80, (7, 6, 5), 3, False),
    ((19, 23, 29), 3, 12, (5, 5, 5), 2, True),
    ((60, 70, 80), 1, 8, (5, 5, 5), 0, True),
], ids=["boxes", "adaptive", "wide", "boxes3d", "rotated", "rotated-large"])
def test_gradients_that_are_not_finite_stay_where_they_belong(spatial, C, R, out, sr, rotated, dtype):
    from medvision_b200 import _C
    nd = len(spatial)
    g = torch.Generator().manual_seed(R)
    rois = _rois(spatial, R, g)
    if rotated:
        lo, hi = rois[:, 1:1 + nd], rois[:, 1 + nd:]
        rois = torch.cat([rois[:, :1], (lo + hi) / 2, hi - lo, torch.rand(R, 1 if nd == 2 else 3, generator=g)], 1)
    rois = rois.to(dtype)
    grad = torch.randn((R, C) + out, generator=g).to(dtype)
    flat = grad.view(-1)
    flat[::997] = float("inf")
    flat[500::1999] = float("nan")
    kw = dict(spatial_scale=1.0, sampling_ratio=sr, aligned=True, order=1, fma_mode=REF_FM if dtype == torch.float32 else 0)
    if rotated:
        kw["trig"] = port.device_trig(rois)
    want = port.backward(grad, rois, (2, C) + spatial, cases.KIND_ROTATED if rotated else cases.KIND_BOX, wide_acc=True, **kw)
    gin = torch.zeros(want.shape, dtype=dtype, device="cuda")
    name = "roi_align_%s%dd_backward" % ("rotated_" if rotated else "", nd)
    getattr(_C, name)(grad.cuda(), rois.cuda(), gin, *out, 1.0, sr, *((True,) if rotated else ()), 1)
    bad = ~torch.isfinite(want)
    assert 0 < int(bad.sum()) < bad.numel() and torch.equal(~torch.isfinite(gin.cpu()), bad)
