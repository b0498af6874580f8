"""Dense 3D calls at the sizes where their kernels change form: axes of one and two voxels, heavy up- and down-sampling, every
roi under a general rotation, more rois than the tables hold.  Forward bit for bit, gradients against the wide-accumulator
restatement."""
import pytest
import torch

import cases
from oracle import port
from util import REF_FM, assert_close, n_mismatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("axes", [1, 3])
@pytest.mark.parametrize("spatial,out,size,R,order", [
    ((1, 20, 33), (8, 24, 24), 1.0, 3, 1),      # one plane: no pair taps
    ((12, 2, 2), (6, 30, 23), 1.2, 3, 1),       # two voxels: every tap next to a border; odd output width
    ((5, 9, 11), (40, 33, 36), 0.6, 2, 1),      # many outputs per voxel
    ((40, 64, 72), (17, 16, 16), 1.4, 3, 1),    # many voxels per output
    ((14, 24, 32), (16, 20, 32), 1.0, 40, 1),   # more rois than the volume's share
    ((14, 24, 32), (16, 20, 32), 1.0, 3, 0),
], ids=["plane", "thin", "up", "down", "rois", "nearest"])
def test_dense_forward_and_gradient(spatial, out, size, R, order, axes, dtype):
    from medvision_b200 import _C
    g = torch.Generator().manual_seed(sum(spatial) + R + axes)
    ext = torch.tensor(spatial[::-1], dtype=torch.float32)
    b = torch.randint(0, 2, (R, 1), generator=g).float()
    centre = ext / 2 + (torch.rand(R, 3, generator=g) - 0.5) * ext * 0.4
    ang = (torch.rand(R, 3, generator=g) - 0.5) * 1.2
    if axes == 1:
        ang[:, :2] = 0
    rois = torch.cat([b, centre, ext * size * (0.8 + 0.4 * torch.rand(R, 3, generator=g)), ang], 1).to(dtype)
    feat = torch.randn((2, 2) + spatial, generator=g).to(dtype)
    kw = dict(spatial_scale=1.0, sampling_ratio=1, aligned=True, order=order, trig=port.device_trig(rois),
              fma_mode=REF_FM if dtype == torch.float32 else 0)
    got = torch.full((R, 2) + out, float("nan"), dtype=dtype, device="cuda")
    _C.affine_3d(feat.cuda(), rois.cuda(), got, *out, 1.0, 1, True, order)
    assert n_mismatch(got, port.forward(feat, rois, out, cases.KIND_ROTATED, **kw)) == 0
    grad = torch.randn((R, 2) + out, generator=g).to(dtype)
    gin = torch.zeros(feat.shape, dtype=dtype, device="cuda")
    _C.roi_align_rotated_3d_backward(grad.cuda(), rois.cuda(), gin, *out, 1.0, 1, True, order)
    want = port.backward(grad, rois, feat.shape, cases.KIND_ROTATED, wide_acc=True, **kw)
    assert_close(gin, want, 2e-3 if dtype == torch.float16 else 2e-5, "gradient")
