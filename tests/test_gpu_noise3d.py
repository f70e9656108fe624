"""The noise variance of a volume against its serial FP32 sum (java/Utils.java:1467-1483),
bit for bit: both round every partial sum, so no tolerance is due. Interiors of one
voxel, of one column, whole numbers of the kernel's 16,384-voxel steps and not, on both
sides of the 65,536 voxels from which the kernel sums; values
that tie on half an ulp, that leap over binades, that are subnormal, zero or not finite."""
import numpy as np
import pytest

from sred_b200 import _lib, utils

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "fp32")


def _values(kind, n, rng):
    v = rng.random(n, dtype=np.float32)
    if kind == "ties":  # squares that are whole multiples of small powers of two
        return np.sqrt(rng.integers(0, 4, n).astype(np.float64) * 0.25).astype(np.float32) * np.float32(2.0 ** -3)
    if kind == "halves":
        return np.where(v < 0.5, np.float32(0.5), np.float32(2.0))
    if kind == "leaps":
        return (v * np.float32(10.0) ** rng.integers(-12, 8, n)).astype(np.float32)
    if kind == "subnormal":
        return v * np.float32(3e-22)
    if kind == "zeros":
        return np.where(v < 0.999, np.float32(0), v).astype(np.float32)
    if kind == "overflow":
        return v * np.float32(5e18)
    if kind == "inf":
        v[n // 2] = np.inf
    if kind == "inf nan":
        v[n // 3] = np.inf
        v[n - 1] = np.nan
    return v


@pytest.mark.parametrize("w,h,d", [(1, 1, 1), (1, 5000, 7), (31, 33, 1), (32, 32, 16), (113, 29, 5), (32, 32, 17),
                                   (17, 1, 1025), (128, 120, 41), (64, 64, 20), (63, 13, 101), (1, 5000, 14),
                                   (64, 128, 10)])
@pytest.mark.parametrize("kind", ["random", "ties", "halves", "leaps", "subnormal", "zeros", "overflow", "inf",
                                  "inf nan"])
def test_noise_variance_3d_bits(ctx, kind, w, h, d):
    rng = np.random.default_rng(w * h + d)
    stds = rng.random((d + 2, h + 4, w + 2), dtype=np.float32)  # the border is not read
    inner = _values(kind, w * h * d, rng)
    stds[1:-1, 2:-2, 1:-1] = inner.reshape(d, h, w)
    with np.errstate(over="ignore", invalid="ignore"):
        total = np.add.accumulate(inner * inner, dtype=np.float32)[-1]
        exp = np.float32(total) / np.float32(w * h * d)
    got = utils.get_relevance_mask_3d(w + 2, h + 4, d + 2, 1, 2, 1, stds.ravel(), 1.0, ctx=ctx).noise_mean_variance
    assert np.array_equal(np.float32(got), exp, equal_nan=True), (float(got), float(exp))
