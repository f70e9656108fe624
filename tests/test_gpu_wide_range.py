"""Denominators and Abs-diff numerators of maps whose weight arguments spread over thousands of
units (bright structures on a nearly silent background): by nodes up to 32,766, whose empty
stretches are stepped over, and pair by pair beyond; Abs-diff by nodes up to 8,190."""
import ctypes as C

import numpy as np
import pytest

from sred_b200 import _lib

pytestmark = pytest.mark.gpu
F = np.float32


def _sums(img, metric):
    import torch
    ctx = _lib.Context(0, "tc")
    h, w = img.shape
    d = torch.from_numpy(img).cuda()
    part = torch.zeros(2 * w * h, dtype=torch.float64, device="cuda")
    info = _lib.RunInfo()
    ctx.check(ctx._L.sred_global_map_2d_shard_sums(ctx.h, metric.encode(), C.c_void_p(d.data_ptr()), w, h, 3, 3, 0.0, 0, 1,
                                                   C.c_void_p(part.data_ptr()), 2 * w * h, None, C.byref(info)), "sums")
    n = int(info.n_relevant - info.n_flat)
    part = part.cpu().numpy()
    return part[:n], part[n:2 * n], info


# One slice of 2,048 blocks and several; the largest a near 1,900, 4,600 to 7,600 (a wide table, Abs-diff
# with and without one), 27,000 to 31,000, and past the table's end.
@pytest.mark.parametrize("w,h", [(40, 36), (130, 97)])
@pytest.mark.parametrize("amp", [1.6, 4.0, 6.4, 26.0, 60.0])
def test_wide_ranges(w, h, amp):
    rng = np.random.default_rng(w)
    img = (1e-6 * rng.random((h, w))).astype(F)
    img[10:22, 12:30] = F(amp) * rng.random((12, 18), dtype=F)
    num, den, info = _sums(img, "Abs. diff. of StdDevs")
    v = np.stack([img[1 + y:h - 1 + y, 1 + x:w - 1 + x] for y, x in ((-1, 0), (0, -1), (0, 0), (0, 1), (1, 0))])
    ws = F(np.sqrt(1.4426950408889634 / np.float64(F(F(info.noise_var) + F(1e-7)))))
    a = (v.astype(np.float64).std(0, ddof=1).ravel() * np.float64(ws)).astype(F).astype(np.float64)
    assert den.size == a.size and a.max() > 1100 * amp
    exp, dnum, slack = np.empty(a.size), np.empty(a.size), np.empty(a.size)
    for i in range(0, a.size, 1024):
        d = np.abs(a[i:i + 1024, None] - a[None])
        wt = np.exp2(-d * d)
        exp[i:i + 1024] = wt.sum(1)
        dnum[i:i + 1024] = (d * wt).sum(1) / np.float64(ws)
        # an argument whose FP32 rounding falls the other way: 2 ln2 d times an ulp of a, half of it for each block
        slack[i:i + 1024] = (wt * 1.4 * d * np.maximum(a[i:i + 1024, None], a[None]) * 2.0 ** -24).sum(1)
    # nodes 6e-11; direct sums: ex2.approx (2^-22), the argument's rounding (at weights that count, 1e-6)
    assert np.all(np.abs(den - exp) <= 2e-6 * exp + slack)
    # pair terms in FP32 from a or from sigma (an ulp of the larger sigma apart), the flush at 2^-126
    sig = a / np.float64(ws)
    ulp = np.array([2.0 ** -23 * np.minimum(np.exp2(-(a - x) ** 2), 1) @ np.maximum(sig, x / np.float64(ws)) for x in a])
    assert np.all(np.abs(num - dnum) <= 6e-6 * dnum + ulp + slack * 12 / np.float64(ws) + 1e-36)
