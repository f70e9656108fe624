"""Abs-diff global maps of images whose block contrasts leave gaps: a block far from all
others, or one of many equal ones, has a numerator as small as its nearest neighbours'
weights, which the sums over all blocks must not drown."""
import ctypes as C

import numpy as np
import pytest

import oracle
from sred_b200 import _lib

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "tc")


def _image(kind, w, h, seed):
    rng = np.random.default_rng(int(10 * seed))
    if kind == "equal":  # a checkerboard's blocks are equal, but for those around three pixels
        y, x = np.mgrid[:h, :w]
        img = (F(8) * ((x + y) & 1)).astype(F)
        for k in range(3):
            img[5 + 7 * k, 3 + 8 * k] += F(60 + seed + 8 * k)
        return img
    img = rng.normal(100, 1, (h, w)).astype(F)
    if kind == "spots":
        for _ in range(6):
            img[rng.integers(2, h - 2), rng.integers(2, w - 2)] += F(rng.uniform(600, 900))
    else:  # two pixels on the border, one block each: a = 100 and `seed` more
        unit = np.sqrt(5 * oracle.mean_noise_var(img) / 1.4426950408889634)
        img[9, 0] += F(unit * 100)
        img[17, w - 1] += F(unit * (100 + seed))
    return img


def _sums(ctx, img):
    import torch
    h, w = img.shape
    d = torch.from_numpy(img).cuda()
    part = torch.zeros(2 * w * h, dtype=torch.float64, device="cuda")
    info = _lib.RunInfo()
    ctx.check(ctx._L.sred_global_map_2d_shard_sums(ctx.h, b"Abs. diff. of StdDevs", C.c_void_p(d.data_ptr()), w, h, 3, 3,
                                                   0.0, 0, 1, C.c_void_p(part.data_ptr()), 2 * w * h, None,
                                                   C.byref(info)), "shard_sums")
    n = int(info.n_relevant - info.n_flat)
    return part.cpu().numpy()[:n], info


# 513 and 1,025 blocks: the last one in order is alone in its slice of 512. Several spots in
# 1,045 and 5,412 blocks; equal blocks in one slice, and in many.
@pytest.mark.parametrize("kind,w,h,seed", [("gap", w, h, g) for w, h in ((29, 21), (27, 43))
                                           for g in (3.0, 4.4, 5.0, 6.0, 7.3, 8.4, 9.5, 10.8)] +
                         [("spots", 57, 21, s) for s in range(4)] + [("spots", 84, 68, s) for s in range(4)] +
                         [("equal", 24, 26, 0), ("equal", 60, 62, 0), ("equal", 60, 62, 7), ("equal", 130, 97, 0)])
def test_isolated_and_equal_blocks(ctx, kind, w, h, seed):
    img = _image(kind, w, h, seed)
    num, info = _sums(ctx, img)
    v = np.stack([img[1 + y:h - 1 + y, 1 + x:w - 1 + x] for y, x in ((-1, 0), (0, -1), (0, 0), (0, 1), (1, 0))])
    ws = F(np.sqrt(1.4426950408889634 / np.float64(F(F(info.noise_var) + F(1e-7)))))
    a = (v.astype(np.float64).std(0, ddof=1).ravel() * np.float64(ws)).astype(F).astype(np.float64)
    assert num.size == a.size
    exp = np.empty(a.size)
    for i in range(0, a.size, 1024):
        d = np.abs(a[i:i + 1024, None] - a[None])
        exp[i:i + 1024] = (d * np.exp2(-d * d)).sum(1) / np.float64(ws)
    # FP32 pair terms: d^2 (half an ulp below 128, times ln 2: 2.7e-6), ex2.approx (2^-22), sums of
    # 32 (1.9e-6), together 4.9e-6; nodes 4e-7, up to 2.5e-6 of terms about to vanish; weights below
    # 2^-126 flush to 0
    np.testing.assert_allclose(num, exp, rtol=5.5e-6, atol=12 * 2.0 ** -126 * a.size / np.float64(ws))
