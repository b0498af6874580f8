"""The native host path: draws made from one array equal the draws made one by one; the ring through which a transform's
rois are uploaded gives every call its own rois, whatever the number of calls in flight, threads and streams."""
import threading

import numpy as np
import pytest
import torch

from medvision_b200.aug_cuda_batch import BatchCudaCropRandomWithAffine, BatchCudaRandomAffine


@pytest.mark.parametrize("shape,patch", [((3, 1, 8, 10, 12), (4, 10, 6)), ((2, 1, 33, 17), (33, 5))])
def test_draws_equal_the_scalar_draws_bit_for_bit(shape, patch):
    dim = len(patch)
    res = {"img_dim": dim, "img": torch.zeros(shape), "img_fields": ["img"], "seg_fields": []}
    t = BatchCudaCropRandomWithAffine(patch, scale=(-0.05, 0.3), shift=0.1, rotate=(5, 5), times=7)
    np.random.seed(3)
    t._forward_params(dict(res))
    state = np.random.get_state()[2]
    np.random.seed(3)
    starts = [t._random_start() for _ in range(7 * shape[0])]
    affine = [([t.get_range(t.scale, 1)] * dim, [t.get_range(t.shift, 0) for _ in range(dim)],
               [np.pi * t.get_range(t.rotate, 0) / 180]) for _ in range(7 * shape[0])]
    assert np.random.get_state()[2] == state
    assert np.array_equal(t.params["start"], np.array([s[::-1] for s in starts]))
    assert np.array_equal(t.params["end"] - t.params["start"], np.broadcast_to(patch[::-1], (7 * shape[0], dim)))
    for k, key in enumerate(("scales", "shifts", "rotate")):
        assert np.array_equal(t.params[key], np.array([a[k] for a in affine]))


@pytest.mark.gpu
def test_roi_uploads_from_several_threads_and_streams_do_not_mix():
    from medvision_b200 import _C
    from medvision_b200.ops import affine_3d
    img = torch.rand(2, 1, 20, 24, 32, generator=torch.Generator().manual_seed(1)).cuda()
    t = BatchCudaRandomAffine(1.0, scale=0.2, shift=0.1, rotate=25)
    sets = []
    for k in range(24):  # three times the ring's slots; one set larger than what the ring was made for
        t._forward_params({"img_dim": 3, "img": img})
        rois = t._rois()
        sets.append(rois.repeat(150, 1) if k == 11 else rois)
    want = [affine_3d(img, r.cuda(), (16, 16, 20), 1.0, 1, True, 1) for r in sets]
    torch.cuda.synchronize()
    got = [None] * len(sets)

    def work(lane):
        with torch.cuda.stream(torch.cuda.Stream()):
            for rep in range(3):
                for k in range(lane, len(sets), 2):
                    got[k] = _C._native.resample_fields(3, [img], [], sets[k], (16, 16, 20), 1, 1)[0][0]

    threads = [threading.Thread(target=work, args=(lane,)) for lane in (0, 1)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    _C.release_cached_memory()  # the ring goes away and comes back
    assert torch.equal(_C._native.resample_fields(3, [img], [], sets[0], (16, 16, 20), 1, 1)[0][0], want[0])


@pytest.mark.gpu
def test_backward_calls_of_several_threads_do_not_disturb_each_other():
    """Box gradients of different shared-memory needs at the same time: every launch succeeds and every gradient is right."""
    from medvision_b200 import _C
    jobs = []
    for k, out in enumerate([(7, 7), (60, 60), (20, 20), (45, 45)]):
        g = torch.Generator().manual_seed(k)
        c = torch.rand(6, 2, generator=g) * 300 + 100
        rois = torch.cat([torch.zeros(6, 1), c - 40, c + 40], 1).cuda()
        jobs.append((torch.randn((6, 1) + out, generator=g).cuda(), rois, out))

    def one(job, gin):
        grad, rois, out = job
        _C.roi_align_2d_backward(grad, rois, gin.zero_(), *out, 1.0, 0, 1)
        return gin

    want = [one(job, torch.empty(1, 1, 512, 512, device="cuda")) for job in jobs]
    torch.cuda.synchronize()
    bad = []

    def work(k):
        try:
            gin = torch.empty(1, 1, 512, 512, device="cuda")
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(1500):
                    one(jobs[k], gin)
                torch.cuda.current_stream().synchronize()
            err = float((gin - want[k]).abs().max() / want[k].abs().max())
            if not err < 1e-5:  # the order of the reductions differs
                bad.append("gradient differs by %g" % err)
        except RuntimeError as e:
            bad.append(str(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad, bad


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["affine", "elastic"])
def test_captured_transforms_keep_their_parameters(kind):
    """A replay gives what the captured call drew, whatever eager calls have done to the upload ring since -- used it over and
    over, grown it, given it back -- and whichever of two graphs goes first."""
    from medvision_b200 import _C
    from medvision_b200.aug_cuda_batch import BatchCudaRandomElasticDeformation
    img = torch.rand(2, 1, 20, 24, 32, generator=torch.Generator().manual_seed(1)).cuda()
    t = (BatchCudaRandomAffine(1.0, scale=0.2, shift=0.1, rotate=25) if kind == "affine"
         else BatchCudaRandomElasticDeformation(1.0, num_control_points=7))
    src = {"img_dim": 3, "img": img, "img_fields": ["img"], "seg_fields": []}

    def call(seed):
        np.random.seed(seed)
        return t(dict(src))["img"]

    want = {seed: call(seed).clone() for seed in (1, 2)}
    assert not torch.equal(want[1], want[2])
    graphs = {}
    for seed in (1, 2):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = call(seed)
        graphs[seed] = graph, out
    for k in range(20):
        call(100 + k)
    big = torch.rand(300, 1, 4, 4, 4).cuda()
    BatchCudaRandomAffine(1.0, scale=0.2, shift=0.1, rotate=25)(dict(src, img=big))  # more rois than the ring was made for
    _C.release_cached_memory()
    for k in range(20):
        call(100 + k)
    for seed in (2, 1, 2):
        graph, out = graphs[seed]
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want[seed])
    del graph, out, graphs   # their memory goes back with the next call
    assert torch.equal(call(1), want[1])
    _C.release_cached_memory()


def test_draws_go_through_the_hooks_of_a_subclass():
    from medvision_b200.aug_cuda_batch import BatchCudaRandomScale

    class Corner(BatchCudaCropRandomWithAffine):
        def _random_start(self):
            return (1, 2, 3)

        @staticmethod
        def get_range(val_range, bias=0, always_pos=False):
            return bias + 0.25

    res = {"img_dim": 3, "img": torch.zeros(2, 1, 8, 10, 12), "img_fields": ["img"], "seg_fields": []}
    t = Corner((4, 5, 6), scale=0.1, shift=0.1, rotate=10, times=3)
    t._forward_params(dict(res))
    assert np.array_equal(t.params["start"], [(3, 2, 1)] * 6) and np.array_equal(t.params["end"], [(9, 7, 5)] * 6)
    assert np.array_equal(t.params["scales"], np.full((6, 3), 1.25)) and np.array_equal(t.params["shifts"], np.full((6, 3), 0.25))
    assert np.array_equal(t.params["rotate"], np.full((6, 1), np.pi * 0.25 / 180))
    t = BatchCudaRandomScale(1.0, 0.1)
    t.get_range = lambda val_range, bias=0, always_pos=False: bias + 0.5  # of the object itself
    t._forward_params(dict(res))
    assert np.array_equal(t.params["scales"], np.full((2, 3), 1.5))
    t = BatchCudaCropRandomWithAffine((4, 5, 6), scale=0.1, shift=0.1, rotate=10)
    t._random_start = lambda: (1, 2, 3)
    t._forward_params(dict(res))
    assert np.array_equal(t.params["start"], [(3, 2, 1)] * 2)


def test_draws_without_numpys_get_bit_generator(monkeypatch):
    """numpy before 1.24"""
    from medvision_b200.aug_cuda_batch import aug_spatial, base
    res = {"img_dim": 3, "img": torch.zeros(2, 1, 8, 10, 12), "img_fields": ["img"], "seg_fields": []}
    t = BatchCudaCropRandomWithAffine((4, 5, 6), scale=0.1, shift=0.1, rotate=10)
    params = []
    for k in range(2):
        if k:
            for module in (base, aug_spatial):
                monkeypatch.setattr(module, "global_bit_generator", base._bit_generator_of_old_numpy)
        np.random.seed(4)
        t._forward_params(dict(res))
        params.append(t.params)
    assert all(np.array_equal(params[0][k], params[1][k]) for k in params[0])


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [True, False])
def test_elastic_deformation_goes_through_the_hooks_of_a_subclass(batched):
    from medvision_b200.aug_cuda import CudaRandomElasticDeformation
    from medvision_b200.aug_cuda_batch import BatchCudaRandomElasticDeformation
    cls = BatchCudaRandomElasticDeformation if batched else CudaRandomElasticDeformation
    shape = (2, 1, 12, 20, 24) if batched else (1, 12, 20, 24)

    class Still(cls):
        def dense_field(self, device):
            return torch.zeros_like(super().dense_field(device))

    class ImageOnly(cls):
        def apply_to_seg(self, result):
            pass

    class Brighter(cls):
        def apply_to_img(self, result):
            super().apply_to_img(result)
            result["img"] = result["img"] + 1

    g = torch.Generator().manual_seed(3)
    img, seg = torch.rand(shape, generator=g).cuda(), torch.randint(0, 4, shape, generator=g, dtype=torch.int32).cuda()

    def call(c):
        np.random.seed(6)
        return c(1.0, num_control_points=7, max_displacement=0.9)({"img_dim": 3, "img": img, "gt_seg": seg, "img_fields": ["img"],
                                                                    "seg_fields": ["gt_seg"]})

    want = call(cls)
    assert not torch.equal(want["img"], img) and not torch.equal(want["gt_seg"], seg)
    got = call(Still)
    assert torch.equal(got["img"], img) and torch.equal(got["gt_seg"], seg)
    got = call(ImageOnly)
    assert torch.equal(got["img"], want["img"]) and got["gt_seg"] is seg
    got = call(Brighter)
    assert torch.equal(got["img"], want["img"] + 1) and torch.equal(got["gt_seg"], want["gt_seg"])
