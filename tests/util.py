"""Shared helpers of the test-suite."""
import os

import numpy as np
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = os.path.join(HERE, "golden", "reference_cuda.npz")

# forward rtol 1e-5 (fp32) / 2e-3 (fp16); fp32 gradients 1e-4 relative.
# A purely relative test is meaningless at zero crossings, so every comparison adds the same
# fraction of the tensor's rms as absolute slack:  |a - b| <= tol * (|b| + rms(b)).
FWD_TOL = {torch.float32: 1e-5, torch.float16: 2e-3, torch.float64: 1e-12}
# Half gradients are accumulated by atomics IN HALF, in whatever order the hardware serves them
# (the reference does the same): two runs of the reference's own kernel differ by several
# half ulps of the running sum, so the half backward bound is that run-to-run spread.
BWD_TOL = {torch.float32: 1e-4, torch.float16: 6e-2, torch.float64: 1e-11}


# float contraction pattern of the reference build (mvr_arith.cuh: kReferenceContraction), for the restatement
REF_FM = 1 | (1 << 1) | (1 << 2) | (1 << 3) | (1 << 5) | (1 << 7) | (1 << 10) | (1 << 13) | \
    (1 << 16) | (1 << 18) | (2 << 20) | (1 << 22)


def bits(t):
    """Integer view for exact comparison (distinguishes nothing but the bit pattern)."""
    t = t.detach().cpu().contiguous()
    return t.view({2: torch.int16, 4: torch.int32, 8: torch.int64}[t.element_size()])


def n_mismatch(a, b):
    a, b = a.detach().cpu(), b.detach().cpu()
    # +0 and -0 compare equal on purpose: no consumer of the op can tell them apart
    return int((a.double() != b.double()).sum())


def assert_close(a, b, tol, what=""):
    a = a.detach().cpu().double()
    b = b.detach().cpu().double()
    assert a.shape == b.shape, (a.shape, b.shape)
    rms = float(b.pow(2).mean().sqrt()) if b.numel() else 0.0
    err = (a - b).abs()
    bound = tol * (b.abs() + rms)
    bad = err > bound
    assert not bool(bad.any()), "%s: %d of %d elements differ beyond tol %g (max abs err %g, rms %g)" % (
        what, int(bad.sum()), a.numel(), tol, float(err.max()), rms)


def load_golden():
    z = np.load(GOLDEN)
    return z


def golden_tensor(z, key, dtype):
    a = z[key]
    t = torch.from_numpy(a.copy())
    if dtype == torch.float16:
        t = t.view(torch.int16).view(torch.float16) if t.dtype != torch.int16 else t.view(torch.float16)
    return t


def assert_half_sums(got, want, grad, rois, kind, adds, trig=None, **kw):
    """``got``: a half gradient that was summed in float and reached memory in at most ``adds`` half additions per roi and element.
    ``want``: the restatement with a wide accumulator.

    A half operation rounds by at most u = 2^-11.  Per element, with S the sum of the contributions' sizes and n its additions:
    the addends are off by some 4 u S (weight products, gradient product, count, the rounding of the addend itself), and every
    addition by u times a partial sum, at most S, in no fixed direction -- together 3.5 sqrt(n) u S, six standard deviations.  Over
    the whole tensor these average out: the error's norm is held to one and a half times its expectation."""
    from oracle import port
    u = 2.0 ** -11
    size = port.backward(grad.abs(), rois, want.shape, kind, trig=trig, wide_acc=True, **kw).double()
    one = torch.ones((1, 1) + tuple(grad.shape[2:]), dtype=torch.half)
    n = torch.zeros((want.shape[0], 1) + tuple(want.shape[2:]), dtype=torch.double)
    for r in range(rois.shape[0]):
        n += port.backward(one, rois[r:r + 1], n.shape, kind, trig=None if trig is None else trig[r:r + 1], wide_acc=True, **kw) != 0
    n *= adds
    err = (got.detach().cpu().double() - want.double()).abs()
    tiny = 2.0 ** -24 * (n + 4)
    over = err > (4 + 3.5 * n.sqrt()) * u * size + tiny
    assert not bool(over.any()), "%d of %d elements are off by more than their additions explain (largest %g)" % (
        int(over.sum()), err.numel(), float(err[over].max()))
    norm = float((((16 + n / 3).sqrt() * u * size + tiny) ** 2).sum().sqrt())
    assert float(err.norm()) <= 1.5 * norm, "error norm %g, expected %g" % (float(err.norm()), norm)
