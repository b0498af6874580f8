"""Sampling kernels with a run-time sample grid (csrc/mvr_flat.cuh) where few outputs are shared by several lanes: eight, four
and two lanes and one, counts that leave the last block partly empty, grids beyond the table of sub-sample offsets, a roi with a
bad batch index.  Forward bit for bit, backward against the wide-accumulator restatement."""
import math

import pytest
import torch

import cases
from oracle import port
from util import REF_FM, assert_close, assert_half_sums, n_mismatch

pytestmark = pytest.mark.gpu

# half additions per roi and voxel: a patch is sent once per slab of the roi's outputs, cells of samples at least half a voxel apart
# at most four times per axis
ADDS = {2: 16, 3: 64}

CASES = [
    # spatial,        channels, rois, output,    sampling, order
    ((37, 41),        3, 9,   (5, 7),    3, 1),
    ((70, 53),        1, 8,   (3, 3),    0, 1),    # up to 20 samples per axis
    ((37, 41),        5, 37,  (7, 7),    3, 0),
    ((70, 53),        9, 31,  (7, 7),    0, 1),
    ((37, 41),        9, 51,  (7, 7),    3, 1),
    ((70, 53),        12, 61, (7, 7),    3, 1),    # one lane again
    ((9, 14, 17),     1, 8,   (3, 2, 5), 3, 1),
    ((19, 23, 29),    3, 9,   (7, 7, 7), 0, 1),
    ((9, 14, 17),     7, 11,  (5, 5, 5), 3, 0),
]


def _rois(spatial, R, g):
    nd = len(spatial)
    ext = torch.tensor(spatial[::-1], dtype=torch.float32)
    b = torch.randint(0, 2, (R, 1), generator=g).float()
    c = torch.rand(R, nd, generator=g) * ext
    s = torch.rand(R, nd, generator=g) * ext * 0.4 + 4.0
    s[1] = ext                        # the whole map
    c[2] = ext * 3                    # outside
    c[3] = ext - 0.5                  # over the border
    a = (torch.rand(R, 1 if nd == 2 else 3, generator=g) * 2 - 1) * math.pi
    return torch.cat([b, c, s, a], 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16], ids=["float32", "float16"])
@pytest.mark.parametrize("spatial,C,R,out,sr,order", CASES,
                         ids=["%s-c%d-%s-s%d-o%d" % ("x".join(map(str, c[0])), c[1], "x".join(map(str, c[3])), c[4], c[5]) for c in CASES])
def test_shared_outputs_match_the_restatement(spatial, C, R, out, sr, order, dtype):
    from medvision_b200 import _C
    nd = len(spatial)
    g = torch.Generator().manual_seed(sum(spatial) + R)
    feat = (torch.rand((2, C) + spatial, generator=g) * 2 - 0.5).to(dtype)
    rois = _rois(spatial, R, g).to(dtype)
    bad = rois.clone()
    bad[6, 0] = 5                     # batch index outside the batch
    fwd, bwd = ((_C.roi_align_rotated_2d_forward, _C.roi_align_rotated_2d_backward) if nd == 2 else
                (_C.roi_align_rotated_3d_forward, _C.roi_align_rotated_3d_backward))
    keep = [i for i in range(R) if i != 6]
    kw = dict(spatial_scale=1.0, sampling_ratio=sr, aligned=True, order=order, trig=port.device_trig(rois[keep]),
              fma_mode=REF_FM if dtype == torch.float32 else 0)
    got = torch.full((R, C) + out, float("nan"), dtype=dtype, device="cuda")
    fwd(feat.cuda(), bad.cuda(), got, *out, 1.0, sr, True, order)
    assert not bool(got[6].any())
    assert n_mismatch(got[keep], port.forward(feat, rois[keep], out, cases.KIND_ROTATED, **kw)) == 0
    grad = torch.randn((R, C) + out, generator=g).to(dtype)
    want = port.backward(grad[keep], rois[keep], feat.shape, cases.KIND_ROTATED, wide_acc=True, **kw)
    gin = torch.zeros(feat.shape, dtype=dtype, device="cuda")
    bwd(grad.cuda(), bad.cuda(), gin, *out, 1.0, sr, True, order)
    if dtype == torch.float32:
        assert_close(gin, want, 1e-5, "gradient")
    else:
        assert_half_sums(gin, want, grad[keep], rois[keep], cases.KIND_ROTATED, ADDS[nd], **kw)
    _C.last_status()


@pytest.mark.parametrize("spatial,C,R,out,sr,order", [
    ((19, 23, 29), 3, 9, (7, 7, 7), 2, 1),      # slabs of a roi
    ((12, 40, 61), 5, 70, (5, 3, 4), 0, 1),     # a roi per block; boxes larger than the shared memory beside small ones
    ((9, 14, 17), 2, 8, (3, 5, 2), 2, 0),
    ((70, 53), 3, 8, (7, 7), 2, 1),
    ((37, 41), 2, 170, (5, 9), 3, 1),
    ((60, 70, 80), 1, 8, (5, 5, 5), 0, 1),      # several blocks per slab
    ((60, 70, 80), 1, 8, (3, 4, 5), 2, 0),
    ((300, 260), 2, 8, (7, 6), 0, 1),
], ids=["slabs", "large", "nearest", "plane", "plane-many", "parts", "parts-sparse", "parts-plane"])
def test_half_gradient_of_rotated_rois(spatial, C, R, out, sr, order):
    from medvision_b200 import _C
    nd = len(spatial)
    g = torch.Generator().manual_seed(sum(spatial) + R)
    rois = _rois(spatial, R, g).half()
    rois[4, 1 + nd:1 + 2 * nd] = 0.3  # far fewer voxels than samples
    grad = torch.randn((R, C) + out, generator=g).half()
    shape = (2, C) + spatial
    kw = dict(spatial_scale=1.0, sampling_ratio=sr, aligned=True, order=order, trig=port.device_trig(rois), fma_mode=0)
    want = port.backward(grad, rois, shape, cases.KIND_ROTATED, wide_acc=True, **kw)
    n = want.numel()
    for offset in (0, 3):             # a gradient tensor at an unaligned place inside a buffer
        buf = torch.full((n + 32,), -0.0, dtype=torch.half, device="cuda")
        gin = buf[16 + offset:16 + offset + n].view(shape)
        gin.zero_()
        (_C.roi_align_rotated_2d_backward if nd == 2 else _C.roi_align_rotated_3d_backward)(
            grad.cuda(), rois.cuda(), gin, *out, 1.0, sr, True, order)
        assert_half_sums(gin, want, grad, rois, cases.KIND_ROTATED, ADDS[nd], **kw)
        around = torch.cat([buf[:16 + offset], buf[16 + offset + n:]])
        assert bool((torch.signbit(around) & (around == 0)).all()), "something was added outside the gradient tensor"


def test_half_gradient_beyond_the_patch_is_as_exact_as_the_flat_kernels():
    """Dense samples in rois larger than the shared-memory patch: summed per cell before they leave.  Against the wide-accumulator
    restatement the flat kernel's error is 1.80e-3 of the gradient's norm, sample by sample it is 2.12e-3."""
    from medvision_b200 import _C
    g = torch.Generator().manual_seed(5)
    R, out = 30, (14, 14, 14)
    rois = torch.cat([torch.zeros(R, 1), torch.rand(R, 3, generator=g) * 48, torch.rand(R, 3, generator=g) * 6 + 24,
                      (torch.rand(R, 3, generator=g) * 2 - 1) * math.pi], 1).half()
    grad = torch.randn((R, 2) + out, generator=g).half()
    want = port.backward(grad, rois, (1, 2, 48, 48, 48), cases.KIND_ROTATED, spatial_scale=1.0, sampling_ratio=4, aligned=True, order=1,
                         trig=port.device_trig(rois), wide_acc=True, fma_mode=0).double()
    gin = torch.zeros((1, 2, 48, 48, 48), dtype=torch.half, device="cuda")
    _C.roi_align_rotated_3d_backward(grad.cuda(), rois.cuda(), gin, *out, 1.0, 4, True, 1)
    assert float((gin.cpu().double() - want).norm() / want.norm()) < 1.9e-3


@pytest.mark.parametrize("rotated,C,R,out,sr,order,dtype", [
    (True, 7, 3100, (7, 7), 1, 1, torch.float32),    # a last group of three channels, a last block partly empty
    (True, 9, 2077, (7, 7), 1, 0, torch.float16),
    (False, 5, 3130, (7, 7), 0, 1, torch.float16),   # a last group of one
    (False, 4, 1601, (14, 14), 3, 1, torch.float16),
    (False, 6, 3130, (7, 7), 0, 1, torch.float32),
], ids=["rotated-float32", "rotated-nearest-float16", "adaptive", "three", "adaptive-float32"])
def test_channel_groups_match_the_restatement(rotated, C, R, out, sr, order, dtype):
    from medvision_b200 import _C
    spatial = (37, 41)
    g = torch.Generator().manual_seed(C * R)
    feat = (torch.rand((2, C) + spatial, generator=g) * 2 - 0.5).to(dtype)
    rois = _rois(spatial, R, g)
    if not rotated:
        rois = torch.cat([rois[:, :1], rois[:, 1:3] - rois[:, 3:5] / 2, rois[:, 1:3] + rois[:, 3:5] / 2], 1)
    rois = rois.to(dtype)
    bad = rois.clone()
    bad[6, 0] = 5
    keep = [i for i in range(R) if i != 6]
    got = torch.full((R, C) + out, float("nan"), dtype=dtype, device="cuda")
    args = (feat.cuda(), bad.cuda(), got) + out + (1.0, sr)
    if rotated:
        _C.roi_align_rotated_2d_forward(*args, True, order)
    else:
        _C.roi_align_2d_forward(*args, order)
    assert not bool(got[6].any())
    want = port.forward(feat, rois[keep], out, cases.KIND_ROTATED if rotated else cases.KIND_BOX, spatial_scale=1.0, sampling_ratio=sr,
                        aligned=True, order=order, trig=port.device_trig(rois[keep]) if rotated else None,
                        fma_mode=REF_FM if dtype == torch.float32 else 0)
    assert n_mismatch(got[keep], want) == 0
    _C.last_status()
