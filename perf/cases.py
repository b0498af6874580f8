"""The calls that users of the framework make, as cases of one benchmark.

Families (key ``op``):
  head     a detection head: RoIAlign / RoIAlignRotated as a module over a feature map, many small rois, a few bins each;
           inference is the forward, training adds the gradient of the features
  dense    RoIAlignRotated over whole volumes with one sample per voxel (differentiable RandomAffine), forward + backward
  crops    affine_2d / affine_3d on device-resident volumes with rois that are on the device: patches cut out of them
  resize   BatchCudaResize on a batch (with or without a label field)
  affine   BatchCudaRandomAffine on a batch with a label field
  crop     BatchCudaCropRandomWithAffine: several patches per volume, image and label field
  elastic  BatchCudaRandomElasticDeformation: dense field from a coarse grid, image and label field
  host     affine_from_host: pinned host volumes in, host patches out

The transforms draw their parameters from numpy's global generator; a pass seeds it first, as a reproducible pipeline
does per step, so that a pass on the same state gives the same result.
"""
import math
import random

import numpy as np
import torch

from medvision_b200.aug_cuda_batch import (BatchCudaCropRandomWithAffine, BatchCudaRandomAffine,
                                           BatchCudaRandomElasticDeformation, BatchCudaResize)
from medvision_b200.ops import RoIAlign, RoIAlignRotated, affine_2d, affine_3d, affine_from_host

DTYPES = {"f16": torch.float16, "f32": torch.float32}
BYTES = {"f16": 2, "f32": 4}


def listed():
    return [
        # inference on a handful of proposals: latency of one call
        dict(name="head3d_infer", op="head", dim=3, rotated=False, dtype="f32", train=False, n=2, c=4, d=64, h=64, w=64,
             rois=16, lo=8.0, hi=48.0, out=7, sampling=2),
        # training step of a 3D detection head (the repository's RoIAlign 3D configuration)
        dict(name="head3d_train", op="head", dim=3, rotated=False, dtype="f32", train=True, n=2, c=4, d=64, h=64, w=64,
             rois=128, lo=8.0, hi=48.0, out=7, sampling=2),
        # training step of a rotated 2D head in half precision (the repository's RoIAlignRotated 2D configuration)
        dict(name="head2d_rot_train", op="head", dim=2, rotated=True, dtype="f16", train=True, n=8, c=3, d=1, h=512, w=512,
             rois=512, lo=16.0, hi=256.0, out=14, sampling=2),
        # the modules' default, adaptive sampling, over a feature map with channels and odd sizes
        dict(name="head2d_adaptive_train", op="head", dim=2, rotated=False, dtype="f32", train=True, n=2, c=32, d=1, h=101,
             w=135, rois=200, lo=8.0, hi=64.0, out=7, sampling=-1),
        # whole CT volumes to the network's input size (the repository's Resize configuration)
        dict(name="resize_ct", op="resize", dim=3, dtype="f16", n=4, c=1, d=160, h=512, w=512, od=128, oh=256, ow=256,
             order=1, seg=False),
        # augmentation of a small batch of volumes with odd sizes, image and label field
        dict(name="affine_odd", op="affine", dim=3, dtype="f16", n=2, c=1, d=79, h=165, w=181, order=1, seg=True),
        # augmentation of a batch of 2D slices with label maps
        dict(name="affine_slices", op="affine", dim=2, dtype="f32", n=16, c=3, d=1, h=512, w=512, order=1, seg=True),
        # differentiable three-axis RandomAffine (the repository's RandomAffine configuration)
        dict(name="dense_train", op="dense", dtype="f16", n=16, c=1, d=128, h=128, w=128, axes=3),
        # patch extraction from eight CT volumes (the repository's crop configuration)
        dict(name="crops_ct", op="crops", dim=3, dtype="f16", n=8, c=1, d=256, h=512, w=512, per=64, pd=96, ph=96, pw=96,
             axes=1, order=1),
        # the batch a segmentation network is fed: patches of image and label from two volumes
        dict(name="crop_batch", op="crop", dim=3, dtype="f16", n=2, c=1, d=128, h=320, w=320, per=4, pd=64, ph=96, pw=96,
             order=1, seg=True),
        # elastic deformation of a batch of CT crops with labels
        dict(name="elastic_ct", op="elastic", dim=3, dtype="f16", n=2, c=1, d=128, h=256, w=256, points=8, seg=True),
        # host volumes in, host patches out
        dict(name="host_crops", op="host", dtype="f16", n=4, c=1, d=128, h=256, w=256, per=16, pd=64, ph=96, pw=96),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["head", "head", "head", "dense", "crops", "resize", "affine", "affine", "crop", "crop", "elastic", "host"])
    dtype = rng.choice(["f16", "f32"])
    if op == "head":
        dim = rng.choice([2, 3])
        out = rng.choice([7, 14] if dim == 2 else [5, 7])
        sampling = rng.choice([2, 2, -1, 1, 3])
        size = [_log(rng, 48, 512) for _ in range(2)] if dim == 2 else [_log(rng, 24, 96) for _ in range(3)]
        hi = rng.uniform(0.3, 0.7) * min(size)
        n, c, rois = rng.randint(1, 4), _log(rng, 1, 64), _log(rng, 8, 800)
        samples = sampling ** dim if sampling > 0 else math.ceil(0.575 * hi / out) ** dim
        while rois * c > 8 and rois * c * out ** dim * max(samples, 16) > 50_000_000:  # a training step's share of proposals and channels
            rois, c = max(8, rois // 2), max(1, c // 2)
        return dict(op="head", dim=dim, rotated=rng.random() < 0.5, dtype=dtype, train=rng.random() < 0.6, n=n, c=c,
                    d=size[0] if dim == 3 else 1, h=size[-2], w=size[-1], rois=rois, lo=round(0.15 * hi, 2), hi=round(hi, 2),
                    out=out, sampling=sampling)
    if op == "dense":
        return dict(op="dense", dtype=dtype, n=rng.randint(1, 8), c=rng.randint(1, 2), d=_log(rng, 32, 128), h=_log(rng, 48, 128),
                    w=_log(rng, 48, 128), axes=rng.choice([1, 3]))
    if op == "crops":
        dim = rng.choice([2, 3, 3])
        d, h, w = (1 if dim == 2 else rng.randint(64, 200)), rng.randint(160, 400), rng.randint(160, 400)
        return dict(op="crops", dim=dim, dtype=dtype, n=rng.randint(1, 4), c=rng.randint(1, 3), d=d, h=h, w=w,
                    per=_log(rng, 1, 32), pd=1 if dim == 2 else rng.randint(24, 64), ph=rng.randint(64, 150),
                    pw=rng.randint(64, 150), axes=rng.choice([1, 1, 3]), order=rng.choice([1, 1, 0]))
    if op == "resize":
        dim = rng.choice([2, 3, 3])
        d, h, w = (1 if dim == 2 else rng.randint(40, 160)), rng.randint(120, 512), rng.randint(120, 512)
        f = [rng.uniform(0.4, 1.4) for _ in range(3)]
        return dict(op="resize", dim=dim, dtype=dtype, n=rng.randint(1, 4), c=rng.randint(1, 2), d=d, h=h, w=w,
                    od=1 if dim == 2 else max(16, int(d * f[0])), oh=int(h * f[1]), ow=int(w * f[2]), order=rng.choice([1, 1, 0]),
                    seg=rng.random() < 0.5)
    if op == "affine":
        dim = rng.choice([2, 3])
        size = [1, _log(rng, 96, 1024), _log(rng, 96, 1024)] if dim == 2 else [_log(rng, 32, 128), _log(rng, 64, 256), _log(rng, 64, 256)]
        return dict(op="affine", dim=dim, dtype=dtype, n=rng.randint(1, 8 if dim == 3 else 16), c=rng.randint(1, 3), d=size[0],
                    h=size[1], w=size[2], order=1, seg=True)
    if op == "crop":
        dim = rng.choice([2, 3, 3])
        d, h, w = (1 if dim == 2 else rng.randint(64, 160)), rng.randint(160, 400), rng.randint(160, 400)
        return dict(op="crop", dim=dim, dtype=dtype, n=rng.randint(1, 4), c=rng.randint(1, 2), d=d, h=h, w=w,
                    per=_log(rng, 1, 16), pd=1 if dim == 2 else rng.randint(24, 64), ph=rng.randint(64, 150),
                    pw=rng.randint(64, 150), order=1, seg=True)
    if op == "elastic":
        dim = rng.choice([2, 3])
        size = [1, _log(rng, 128, 1024), _log(rng, 128, 1024)] if dim == 2 else [_log(rng, 32, 128), _log(rng, 96, 256), _log(rng, 96, 256)]
        return dict(op="elastic", dim=dim, dtype=dtype, n=rng.randint(1, 4), c=rng.randint(1, 2), d=size[0], h=size[1],
                    w=size[2], points=rng.randint(6, 10), seg=True)
    return dict(op="host", dtype=dtype, n=rng.randint(1, 4), c=1, d=rng.randint(64, 128), h=rng.randint(128, 256),
                w=rng.randint(128, 256), per=_log(rng, 2, 24), pd=rng.randint(24, 64), ph=rng.randint(64, 112), pw=rng.randint(64, 112))


# ---- inputs -------------------------------------------------------------------------------------

def _spatial(case):
    return (case["d"], case["h"], case["w"]) if case.get("dim", 3) == 3 else (case["h"], case["w"])


def _patch(case):
    return (case["pd"], case["ph"], case["pw"]) if case.get("dim", 3) == 3 else (case["ph"], case["pw"])


def _ct(shape, dtype, g):
    """CT-like values: ~N(-300, 400) clipped to [-1024, 3071], whole numbers, scaled to [0, 1]."""
    v = torch.empty(shape, device="cuda").normal_(-300, 400, generator=g).round_().clamp_(-1024, 3071)
    return v.add_(1024).div_(4095).to(dtype)


def _smooth(shape, dtype, g):
    """A smooth random field of unit deviation: coarse noise, interpolated."""
    coarse = [max(2, s // 8) for s in shape[2:]]
    x = torch.randn(shape[:2] + tuple(coarse), device="cuda", generator=g)
    x = torch.nn.functional.interpolate(x, size=shape[2:], mode="trilinear" if len(shape) == 5 else "bilinear", align_corners=True)
    return (x / x.std()).to(dtype)


def _labels(shape, g):
    """Label maps of a few connected regions (five classes), int32."""
    return (_smooth((shape[0], 1) + shape[2:], torch.float32, g) * 1.5 + 2).round_().clamp_(0, 4).int()


def _head_rois(case, dtype, g):
    r, dim = case["rois"], case["dim"]
    ext = torch.tensor([case["w"], case["h"], case["d"]][:dim], device="cuda", dtype=torch.float32)
    b = torch.randint(0, case["n"], (r, 1), device="cuda", generator=g).float()
    c = torch.rand(r, dim, device="cuda", generator=g) * ext
    s = torch.rand(r, dim, device="cuda", generator=g) * (case["hi"] - case["lo"]) + case["lo"]
    if not case["rotated"]:
        return torch.cat([b, c - s / 2, c + s / 2], 1).to(dtype)
    a = (torch.rand(r, 1 if dim == 2 else 3, device="cuda", generator=g) * 2 - 1) * math.pi
    return torch.cat([b, c, s, a], 1).to(dtype)


def _angles(case, r, g, deg):
    dim = case.get("dim", 3)
    a = (torch.rand(r, 1 if dim == 2 else 3, device="cuda", generator=g) * 2 - 1) * math.radians(deg)
    if dim == 3 and case.get("axes", 1) == 1:
        a[:, :2] = 0
    return a


def _crop_rois(case, g):
    """Patches at random places inside the volumes, turned by up to 20 degrees, scaled by 0.9-1.1."""
    size, patch = _spatial(case), _patch(case)
    r, dim = case["n"] * case["per"], len(size)
    ext = torch.tensor(size[::-1], device="cuda", dtype=torch.float32)
    p = torch.tensor(patch[::-1], device="cuda", dtype=torch.float32)
    b = torch.arange(case["n"], device="cuda").repeat_interleave(case["per"]).float().view(-1, 1)
    scale = torch.rand(r, 1, device="cuda", generator=g) * 0.2 + 0.9
    start = torch.rand(r, dim, device="cuda", generator=g) * (ext - p)
    return torch.cat([b, start + p / 2, p / scale, _angles(case, r, g, 20)], 1)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype, op = DTYPES[case["dtype"]], case["op"]
    size = _spatial(case)
    shape = (case["n"], case["c"]) + size
    if op == "head":
        x = torch.randn(shape, device="cuda", generator=g).to(dtype)
        rois = _head_rois(case, dtype, g)
        out = (case["out"],) * case["dim"]
        module = (RoIAlignRotated if case["rotated"] else RoIAlign)(out, 1.0, case["sampling"])
        grad = torch.randn((case["rois"], case["c"]) + out, device="cuda", generator=g).to(dtype) if case["train"] else None
        return dict(op=op, module=module, x=x.requires_grad_(case["train"]), rois=rois, grad=grad)
    if op == "dense":
        x = _smooth(shape, dtype, g).requires_grad_(True)
        n, ext = case["n"], torch.tensor(size[::-1], device="cuda", dtype=torch.float32)
        scale = torch.rand(n, 1, device="cuda", generator=g) * 0.4 + 0.8
        shift = (torch.rand(n, 3, device="cuda", generator=g) * 2 - 1) * 10
        rois = torch.cat([torch.arange(n, device="cuda").float().view(-1, 1), ext / 2 - shift / scale, ext / scale,
                          _angles(case, n, g, 30)], 1).to(dtype)
        grad = torch.randn(shape, device="cuda", generator=g).to(dtype)
        return dict(op=op, module=RoIAlignRotated(size, 1.0, sampling_ratio=1), x=x, rois=rois, grad=grad)
    if op == "crops":
        return dict(op=op, x=_ct(shape, dtype, g), rois=_crop_rois(case, g).to(dtype), patch=_patch(case), order=case["order"])
    if op == "host":
        x = torch.empty(shape, dtype=dtype, pin_memory=True)
        x.copy_(_ct(shape, dtype, g))
        return dict(op=op, x=x, rois=_crop_rois(case, g).cpu(), patch=_patch(case))
    result = {"img_dim": case["dim"], "img": _ct(shape, dtype, g), "img_fields": ["img"], "seg_fields": []}
    if case["seg"]:
        result.update(gt_seg=_labels(shape, g), seg_fields=["gt_seg"])
    if op == "resize":
        target = (case["od"], case["oh"], case["ow"])[3 - case["dim"]:]
        t = BatchCudaResize(scale=target, order=case["order"])
    elif op == "affine":
        t = BatchCudaRandomAffine(1.0, scale=0.2, shift=0.1, rotate=25, order=case["order"])
    elif op == "crop":
        t = BatchCudaCropRandomWithAffine(_patch(case), scale=0.1, shift=0.05, rotate=20, order=case["order"], times=case["per"])
    else:
        t = BatchCudaRandomElasticDeformation(1.0, num_control_points=case["points"], max_displacement=0.8)
    return dict(op="augment", transform=t, result=result, seed=seed % (1 << 31))


def run(state):
    op = state["op"]
    if op == "augment":
        np.random.seed(state["seed"])
        random.seed(state["seed"])
        result = dict(state["result"])
        result = state["transform"](result)
        return {k: result[k] for k in result["img_fields"] + result["seg_fields"]}
    if op == "crops":
        fn = affine_2d if len(state["patch"]) == 2 else affine_3d
        return fn(state["x"], state["rois"], state["patch"], 1.0, 1, True, state["order"])
    if op == "host":
        return affine_from_host(state["x"], state["rois"], state["patch"], 1.0, 1, True, 1)
    out = state["module"](state["x"], state["rois"])
    if state["grad"] is None:
        return out
    return out, torch.autograd.grad(out, state["x"], state["grad"])[0]


# ---- what a pass cannot do without ----------------------------------------------------------------

def work(case):
    op, e = case["op"], BYTES[case["dtype"]]
    size = _spatial(case)
    vol = math.prod(size)
    dim = len(size)
    feat = case["n"] * case["c"] * vol
    if op == "head":
        out = case["rois"] * case["c"] * case["out"] ** dim
        mean = (case["lo"] + case["hi"]) / 2
        samples = case["sampling"] ** dim if case["sampling"] > 0 else math.ceil(mean / case["out"]) ** dim
        read = min(feat, case["rois"] * case["c"] * mean ** dim)  # a proposal's extent, no more than the map
        flops = out * samples * 2 * 2 ** dim
        if not case["train"]:
            return dict(bytes=e * (read + out), flops=flops)
        return dict(bytes=e * (read + out + out + feat), flops=2 * flops)
    if op == "dense":
        return dict(bytes=e * 4 * feat, flops=feat * 2 * 16)
    label_in = label_out = 0
    if op == "resize":
        out = case["n"] * case["c"] * (case["od"] if dim == 3 else 1) * case["oh"] * case["ow"]
        seen = 1.0
        if case["seg"]:
            label_in, label_out = case["n"] * vol, out // case["c"]
    elif op in ("affine", "elastic"):
        out, seen = feat, 1.0
        label_in = label_out = case["n"] * vol
    else:
        patch = math.prod(_patch(case))
        out = case["n"] * case["per"] * case["c"] * patch
        seen = 1.0 - math.exp(-case["per"] * patch / vol)  # share of a volume that random patches cover
        if op == "host":
            seen = 1.0  # the volumes go up whole
        if case.get("seg"):
            label_in, label_out = seen * case["n"] * vol, out // case["c"]
    return dict(bytes=e * (seen * feat + out) + 4 * (label_in + label_out), flops=out * 2 * 2 ** dim)


def tolerance(case):
    half = case["dtype"] == "f16"
    if case["op"] == "elastic":
        # the last bits of the displacement move a sample position by a rounding step of the image's type, and a label
        # to the neighbouring voxel where the position is a tie
        return {"rel": 5e-3 if half else 1e-4, "max": 0.9 if half else 1e-2, "differ": 1e-3}
    if case["op"] == "head" and case["train"]:
        return {"rel": 1e-2 if half else 1e-5}  # half gradients are summed in half, in no fixed order
    return {"rel": 2e-3 if half else 1e-5}
