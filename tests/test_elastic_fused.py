"""The elastic deformation straight from the coarse grid against its two-step form (dense field by affine_*(order 3), then
apply_offset_*): the same displacement field to float rounding, and the bits of the warp by that field."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [
    # shape,               dtype,         label,       control points
    ((2, 1, 9, 17, 64),    torch.float16, torch.int32, 8),
    ((1, 3, 5, 70, 33),    torch.float32, torch.uint8, (4, 7, 9)),    # odd width, the smallest grid, several channels
    ((3, 2, 1, 8, 1),      torch.float32, torch.int16, 6),            # single voxels along two axes
    ((1, 1, 64, 96, 130),  torch.float16, torch.int64, (10, 12, 20)),
    ((2, 3, 50, 67),       torch.float32, torch.int32, 7),            # 2D
    ((1, 1, 129, 258),     torch.float16, torch.int32, (9, 33)),
    ((1, 1, 8, 40, 40),    torch.float32, torch.int32, (6, 60, 60)),  # tables exceed shared memory: two-step form
]


@pytest.mark.parametrize("shape,dtype,label,points", CASES, ids=["x".join(map(str, c[0])) for c in CASES])
def test_fused_warp_equals_the_two_steps(shape, dtype, label, points):
    from medvision_b200.aug_cuda_batch import BatchCudaRandomElasticDeformation
    from medvision_b200.ops import affine_2d, affine_3d
    dim = len(shape) - 2
    g = torch.Generator().manual_seed(sum(shape))
    img = torch.rand(shape, generator=g).to(dtype).cuda()
    seg = torch.randint(0, 200, (shape[0], 2) + shape[2:], generator=g).to(label).cuda()
    res = {"img_dim": dim, "img": img, "gt_seg": seg, "img_fields": ["img"], "seg_fields": ["gt_seg"]}
    np.random.seed(4)
    t = BatchCudaRandomElasticDeformation(1.0, num_control_points=points, max_displacement=0.9)
    out = t(res)
    dense = t.dense_field(img.device)
    coarse = (torch.from_numpy(t.params).permute(0, dim + 1, *range(1, dim + 1)) / 2).contiguous()
    grid = coarse.shape[2:]
    rois = torch.tensor([[b] + [s / 2 for s in grid[::-1]] + [s - 3. for s in grid[::-1]] + [0.] * (1 if dim == 2 else 3)
                         for b in range(shape[0])])
    fn = affine_2d if dim == 2 else affine_3d
    want = fn(coarse.cuda(), rois.cuda(), tuple(shape[2:]), 1.0, 1, True, 3)
    torch.testing.assert_close(dense, want, rtol=1e-5, atol=1e-6 * float(coarse.abs().max()))
    assert torch.equal(out["img"], t.elastic_transform(img))
    assert out["gt_seg"].dtype == torch.int32 and torch.equal(out["gt_seg"], t.elastic_transform(seg, order=0))
    # label alone
    t.tmp_params = None
    alone = t._warp_fields([], [seg])[1][0]
    assert torch.equal(alone, out["gt_seg"])
