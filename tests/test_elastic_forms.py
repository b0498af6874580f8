"""Elastic deformation of an image and its labels straight from the coarse grid, at the sizes where its kernel changes form (a table
along w, taps at fixed distances, several channels): the same bits as the warp by the dense field."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("shape,C,label", [
    ((2, 2, 2), 1, torch.uint8),         # every tap next to a border
    ((1, 40, 30), 1, torch.int32),       # one plane: no fixed distances
    ((48, 300, 65), 1, torch.int16),     # the table, odd width
    ((48, 300, 64), 1, torch.int64),
    ((48, 300, 64), 2, torch.int32),     # several channels: no table
    ((3, 3, 2049), 1, torch.int32),      # the longest row of fixed distances
    ((3, 3, 2050), 1, torch.int32),
    ((15000, 62), 1, torch.int32),       # the table without fixed distances
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_forms_equal_the_warp_by_the_dense_field(shape, C, label, dtype):
    from medvision_b200.aug_cuda_batch import BatchCudaRandomElasticDeformation
    g = torch.Generator().manual_seed(sum(shape) + C)
    img = torch.randn((2, C) + shape, generator=g).to(dtype).cuda()
    seg = torch.randint(0, 200, (2, C) + shape, generator=g).to(label).cuda()
    if label in (torch.int32, torch.int64):
        seg[..., ::2] += 2001  # beyond the consecutive integers of half
    res = {"img_dim": len(shape), "img": img, "gt_seg": seg, "img_fields": ["img"], "seg_fields": ["gt_seg"]}
    np.random.seed(6)
    t = BatchCudaRandomElasticDeformation(1.0, num_control_points=7, max_displacement=0.9)
    out = t(res)
    assert torch.equal(out["img"], t.elastic_transform(img))
    assert torch.equal(out["gt_seg"], t.elastic_transform(seg, order=0))
