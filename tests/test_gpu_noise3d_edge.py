"""The noise variance of a volume where a square is 4194303.75 units of the sum's last place:
sigma = sqrt(0.5) in FP32 squares to an all-ones mantissa, and three of them sum to just below
1.5. Serial FP32 sums, bit for bit (no tolerance is due), on both sides of the 65,536 voxels from
which the device sums."""
import numpy as np
import pytest

from sred_b200 import _lib, utils

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "fp32")


# The fourth such voxel in the run of 16 of the first three, in the next one, in another warp's,
# in the kernel's second step of 16,384; at three binades; between zeros, between small values,
# and everywhere.
@pytest.mark.parametrize("at", [3, 17, 600, 8191, 16389, 40000])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20, 2.0 ** 18])
@pytest.mark.parametrize("d", [10, 41])
@pytest.mark.parametrize("rest", ["zeros", "small", "constant"])
def test_all_ones_square(ctx, at, scale, d, rest):
    w, h = 64, 80
    n = w * h * d
    v = F(np.sqrt(F(0.5)))
    inner = np.zeros(n, F)
    if rest == "small":
        inner = np.random.default_rng(at).random(n, dtype=F) * F(2.0 ** -14)
        inner[:at + 1] = 0
    if rest == "constant":
        inner[at:] = v
    inner[[0, 1, 2, at]] = v
    inner *= F(scale)
    stds = np.zeros((d + 2, h + 2, w + 2), F)
    stds[1:-1, 1:-1, 1:-1] = inner.reshape(d, h, w)
    exp = np.add.accumulate(inner * inner, dtype=F)[-1] / F(n)
    got = utils.get_relevance_mask_3d(w + 2, h + 2, d + 2, 1, 1, 1, stds.ravel(), 1.0, ctx=ctx).noise_mean_variance
    assert F(got) == exp, (float(got), float(exp))
