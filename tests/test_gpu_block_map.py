"""The 2D block map against the same operations in numpy FP32, bit for bit: the kernels
follow the reference's evaluation order with every operation rounded
(cl/kernelGetBlock{Pearson,Ssim,Nrmse,AbsDiffStds}2D.cl, java/CLUtils.java:788-960),
so no tolerance is due. Sizes: both widths of the launch rule, widths with and without
remainders of 4, 32 and 128, several frames, a tall block whose tile exceeds 48 KB."""
import numpy as np
import pytest

from sred_b200 import _lib, clutils, utils

pytestmark = pytest.mark.gpu
F = np.float32
EPS = F(1e-7)


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "fp32")


def _offsets(bw, bh):
    rw, rh = bw // 2, bh // 2
    return [(dy, dx) for dy in range(-rh, rh + 1) for dx in range(-rw, rw + 1)
            if F(dx * dx) / F(rw * rw) + F(dy * dy) / F(rh * rh) <= F(1)]


def _reference(img, offs, bw, bh, y, x):
    px = np.array([img[y + dy, x + dx] for dy, dx in offs], F)
    m = F(px.mean())
    px = px - m
    sd = F(np.sqrt((px.astype(np.float64) ** 2).sum() / (px.size - 1)))
    return utils.ReferenceBlock2D(px, bw, bh, bw // 2, bh // 2, px.size, m, sd)


def _expected(metric, img, ref, offs, rw, rh, normalize):
    h, w = img.shape
    ih, iw = h - 2 * rh, w - 2 * rw
    win = [img[rh + dy:rh + dy + ih, rw + dx:rw + dx + iw] for dy, dx in offs]
    k = F(len(offs))
    mean = np.zeros((ih, iw), F)
    for v in win:
        mean = mean + v
    mean = mean / k
    var, acc = np.zeros((ih, iw), F), np.zeros((ih, iw), F)
    for p, v in zip(ref.pixels, win):
        d = v - mean
        var = var + d * d
        t = p - d
        acc = acc + (t * t if metric.startswith("NRMSE") else p * d)
    sd = np.sqrt(var / (k - F(1)))
    rs, rm = F(ref.std), F(ref.mean)
    if metric.startswith("Abs"):
        m = np.abs(rs - sd)
        m = F(1) - (m - m.min()) / (max(m.max(), F(1.4e-45)) - m.min() + EPS)
    elif metric.startswith("NRMSE"):
        m = np.sqrt(acc / k)
        m = (m - m.min()) / (m.max() - m.min() + EPS)
        with np.errstate(divide="ignore"):
            m = np.where(m == 0, F(1), F(1) / m)
    else:
        cov = acc / (k - F(1))
        if metric == "SSIM":
            a = F(2) * rm * mean + F(0.0001)
            b = F(2) * cov + F(0.0009)
            m = np.maximum(F(0), a * b / ((rm * rm + mean * mean + F(0.0001)) * (rs * rs + sd * sd + F(0.0009))))
        else:
            m = np.maximum(F(0), cov / (rs * sd + EPS))
    if normalize:
        m = (m - m.min()) / (m.max() - m.min() + EPS)
    out = np.zeros((h, w), F)
    out[rh:h - rh, rw:w - rw] = m
    return out


@pytest.mark.parametrize("w,h,frames,bw,bh", [(9, 7, 1, 3, 3), (33, 34, 2, 5, 7), (129, 65, 1, 7, 3), (20, 420, 1, 3, 401),
                                              (520, 910, 1, 5, 5), (517, 301, 3, 3, 9), (130, 97, 40, 3, 3)])
@pytest.mark.parametrize("metric", ["Pearson's R", "SSIM", "NRMSE (inverted)", "Abs. Diff. of StdDevs."])
def test_block_map_bits(ctx, metric, w, h, frames, bw, bh):
    import torch
    rng = np.random.default_rng(w * h)
    img = (rng.random((frames, h, w), dtype=F) * F(100)).astype(F)
    offs = _offsets(bw, bh)
    ref = _reference(img[0], offs, bw, bh, h // 2, w // 2)
    d_in = torch.from_numpy(img).cuda()
    d_out = torch.empty_like(d_in)
    for normalize in (False, True):
        clutils.block_map_device(metric, d_in.data_ptr(), w, h, frames, ref, 0.0, normalize, d_out.data_ptr(), ctx=ctx)
        got = d_out.cpu().numpy()
        for f in range(frames):
            exp = _expected(metric, img[f], ref, offs, bw // 2, bh // 2, normalize)
            assert np.array_equal(got[f], exp), (f, normalize, float(np.abs(got[f] - exp).max()))


@pytest.mark.parametrize("w,h,d,bw,bh,bd", [(37, 9, 5, 5, 3, 3), (38, 10, 6, 5, 5, 3), (69, 9, 8, 5, 3, 7), (70, 11, 5, 5, 3, 3),
                                            (133, 17, 4, 3, 5, 3), (260, 9, 9, 9, 7, 5), (9, 9, 9, 9, 3, 3)])
@pytest.mark.parametrize("metric", clutils.BLOCK_METRICS)
def test_block_map_3d_bits(ctx, metric, w, h, d, bw, bh, bd):
    """Interiors of 33, 34, 65, 66, 131 and 252 columns (windows of 2 and 4, whole and ragged
    last ones, two tiles) and of one; with and without normalisation and relevance mask."""
    import oracle
    rng = np.random.default_rng(w + h)
    vol = rng.random((d, h, w), dtype=F)
    z, y, x = d // 2, h // 2, w // 2
    rb = utils.get_reference_block_3d(vol[z - bd // 2:z + bd // 2 + 1, y - bh // 2:y + bh // 2 + 1,
                                          x - bw // 2:x + bw // 2 + 1])
    for c, normalize in ((0.0, True), (0.0, False), (1.0, True)):
        exp = oracle.block_map3d(metric, vol, rb.pixels, bw, bh, bd, rb.mean, rb.std, c, normalize)["map"]
        got = clutils.calculate_block_repetition_map_3d(metric, utils.InputImage3D(vol.ravel(), w, h, d), rb, c, normalize,
                                                        ctx=ctx)
        assert np.array_equal(got, exp.ravel(), equal_nan=True), (c, normalize)
