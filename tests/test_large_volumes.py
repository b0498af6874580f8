"""Float channels of 2^30 to 2^31 elements (1024^3 is one), whose offsets do not fit 32 bits as bytes: the dense forwards and the
displacement-field warp keep their own kernels there, and give what the general path gives.  The samples lie at both ends of the
volume, so that offsets on either side of 4 GiB occur."""
import pytest
import torch

import cases
from oracle import port
from util import REF_FM

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def elements():
    # noise of an odd period: an offset that is wrong by 4 GiB finds another value
    noise = torch.rand((1 << 27) + 1, generator=torch.Generator().manual_seed(7)).repeat(9)
    return noise, noise.cuda()


def _kernels(fn):
    """Names of the kernels that ``fn`` launches, from a CUDA graph."""
    from cuda.bindings import driver, runtime
    fn()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        out = fn()
    raw = graph.raw_cuda_graph()
    _, _, n = runtime.cudaGraphGetNodes(raw, 0)
    _, nodes, n = runtime.cudaGraphGetNodes(raw, n)
    names = []
    for node in nodes[:n]:
        if runtime.cudaGraphNodeGetType(node)[1] != runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel:
            continue
        err, par = driver.cuGraphKernelNodeGetParams(driver.CUgraphNode(int(node)))
        assert err == driver.CUresult.CUDA_SUCCESS
        err, name = driver.cuFuncGetName(par.func) if int(par.func) else driver.cuKernelGetName(par.kern)
        assert err == driver.CUresult.CUDA_SUCCESS
        names.append(name.decode())
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    return names, out


def _rois(spatial, kind):
    """Patches at both ends of the volume and one that samples every fourth voxel (a footprint beyond the staged boxes)."""
    nd = len(spatial)
    ext = torch.tensor(spatial[::-1], dtype=torch.float32)
    centre = torch.stack([torch.full((nd,), 20.0), ext - 17.3, ext - 70, ext / 2])
    size = torch.tensor([30.0, 36.0, 130.0, 28.0]).view(-1, 1).repeat(1, nd)
    if kind == "box":
        return torch.cat([torch.zeros(4, 1), centre - size / 2, centre + size / 2], 1)
    ang = torch.tensor([0.3, -0.4, 0.2, 0.5]).view(-1, 1)
    if nd == 3:
        ang = torch.cat([ang * 0.5, -ang, ang], 1)
        if kind == "z":
            ang[:, :2] = 0
        elif kind == "mixed":
            ang[::2, :2] = 0
    return torch.cat([torch.zeros(4, 1), centre, size, ang], 1)


@pytest.mark.parametrize("spatial,out,kind,kernel", [
    ((1024, 1024, 1024), (8, 32, 32), "mixed", "stream3d"),     # both launches
    ((1024, 1024, 1024), (8, 32, 32), "box", "stream3d_tma"),
    ((1057, 1001, 1021), (8, 32, 31), "z", "stream3d"),         # no tensor map: rows of no whole 16 bytes
    ((1057, 1001, 1021), (8, 32, 31), "xyz", "stream3d"),
    ((32768, 32800), (64, 66), "xyz", "plane2d"),
], ids=["rotated", "box", "odd-z", "odd-xyz", "plane"])
def test_dense_forward_keeps_its_kernel(elements, spatial, out, kind, kernel):
    from medvision_b200.ops import RoIAlign, affine_2d, affine_3d
    n = 1
    for s in spatial:
        n *= s
    assert 2 ** 30 <= n < 2 ** 31
    host, x = (e[:n].view((1, 1) + spatial) for e in elements)
    rois = _rois(spatial, kind).cuda()

    def call(r=rois):
        if kind == "box":
            return RoIAlign(out, 1.0, 1)(x, r)
        return (affine_2d if len(spatial) == 2 else affine_3d)(x, r, out, 1.0, 1, True, 1)

    names, got = _kernels(call)
    assert names and all(kernel in k for k in names), names
    want = port.forward(host, rois.cpu(), out, cases.KIND_BOX if kind == "box" else cases.KIND_ROTATED, spatial_scale=1.0,
                        sampling_ratio=1, aligned=True, order=1, trig=None if kind == "box" else port.device_trig(rois.cpu()),
                        fma_mode=REF_FM)
    assert torch.equal(got.cpu(), want)


def test_offset_warp_keeps_its_kernel(elements):
    from medvision_b200.ops import apply_offset_3d
    spatial = (1030, 1024, 1024)
    n = spatial[0] * spatial[1] * spatial[2]
    x = elements[1][:n].view((1, 1) + spatial)
    # multiples of a quarter voxel: positions and weights are exact, wherever a slab starts
    field = torch.randint(-12, 13, (1, 3) + spatial, device="cuda", dtype=torch.int8).float().div_(4)
    names, got = _kernels(lambda: apply_offset_3d(x, field, 1))
    # template arguments: element type, axes, voxel by voxel, 64-bit offsets
    assert any("apply_offset_kernelIfLi3ELb0ELb1E" in k for k in names), names
    for lo in (0, spatial[0] - 20):  # slabs at either end, through the form for small volumes
        slab = slice(lo, lo + 20)
        small = apply_offset_3d(x[:, :, slab].contiguous(), field[:, :, slab].contiguous(), 1)
        inner = slice(0, 16) if lo == 0 else slice(4, 20)  # samples that stay inside the slab, or leave the volume with it
        assert torch.equal(got[:, :, slab][:, :, inner], small[:, :, inner])
