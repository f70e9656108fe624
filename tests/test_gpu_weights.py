"""The parts of the global map that carry the weights: the denominators as one
function of one variable, the order of the blocks, the factorised pair loop in
each of its forms, and the split-FP16 operand at every block count of K."""
import ctypes as C

import numpy as np
import pytest

import oracle
from sred_b200 import _lib, clutils, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "tc")


def _sums(ctx, engine, img, b, relc, metric="Pearson's R"):
    """num and den of the unsharded map and the run info (shard 0 of 1)."""
    import torch
    ctx.set_engine(engine)
    h, w = img.shape
    d = torch.from_numpy(img).cuda()
    part = torch.zeros(2 * w * h, dtype=torch.float64, device="cuda")
    info = _lib.RunInfo()
    ctx.check(ctx._L.sred_global_map_2d_shard_sums(ctx.h, metric.encode(), C.c_void_p(d.data_ptr()), w, h, b, b, relc, 0,
                                                   1, C.c_void_p(part.data_ptr()), 2 * w * h, None, C.byref(info)),
              "shard_sums")
    n = int(info.n_relevant - info.n_flat)
    part = part.cpu().numpy()
    return part[:n], part[n:2 * n], info


def _expected_a(img, b, info):
    """FP32 stds and weight arguments of the listed blocks, raster order."""
    r = b // 2
    _, s32 = oracle.local_stats(img, b, b)
    h, w = img.shape
    offs = [(y, x) for y in range(-r, r + 1) for x in range(-r, r + 1)
            if np.float32(x * x) / np.float32(r * r) + np.float32(y * y) / np.float32(r * r) <= 1]
    v = np.stack([img[r + y:h - r + y, r + x:w - r + x] for y, x in offs]).astype(np.float64)
    s64 = v.std(0, ddof=1)
    s = s32[r:h - r, r:w - r]
    use = ~(s * s < np.float32(info.threshold)) & (s != 0)
    ws = np.float32(np.sqrt(1.4426950408889634 / np.float64(np.float32(np.float32(info.noise_var) + np.float32(1e-7)))))
    return s[use], (s64[use] * np.float64(ws)).astype(np.float32)


def _weights_image(w, h, bright):
    if not bright:
        return synth.normalize_input(synth.spot_image(w, h, 4, seed=w))
    rng = np.random.default_rng(5)
    img = (1e-6 * rng.random((h, w))).astype(np.float32)
    img[40:60, 40:70] = 4 * rng.random((20, 30), dtype=np.float32)
    return img


# Images whose listed blocks number one slice of 2,048 or less, a slice and a few, several
# slices, and enough to be sorted; and with a bright square on a nearly silent background (the a-range beyond the
# node table: direct sums).
@pytest.mark.parametrize("w,h,b,bright", [(21, 19, 3, 0), (50, 46, 5, 0), (130, 97, 9, 0), (150, 140, 5, 1), (184, 170, 3, 0)])
@pytest.mark.parametrize("engine", ["tc", "fp32"])
def test_denominators_and_block_order(ctx, engine, w, h, b, bright):
    img = _weights_image(w, h, bright)
    _, den, info = _sums(ctx, engine, img, b, 0.0)
    s, a = _expected_a(img, b, info)
    assert den.size == a.size
    if bright:
        assert a.max() > 2046, a.max()
    # from 28,000 blocks on by the top 22 bits below the sign of the FP32 std, ties in raster order
    if engine == "tc" and a.size >= 28000:
        a = a[np.argsort(s.view(np.uint32) >> 9, kind="stable")]
    a = a.astype(np.float64)
    exp = np.concatenate([np.exp2(-(a[i:i + 1024, None] - a[None]) ** 2).sum(1) for i in range(0, a.size, 1024)])
    # nodes: 6e-11 relative, plus an FP32 rounding of an argument that falls the other way
    # (2 ln2 d da 2^-24, below 1e-6); direct sums: ex2.approx (2^-22) and FP32 arguments
    np.testing.assert_allclose(den, exp, rtol=4e-6 if bright else 1e-6)


# The same sizes; the slices of Abs-diff hold 512 blocks.
@pytest.mark.parametrize("w,h,b", [(21, 19, 3), (34, 18, 3), (50, 46, 5), (130, 97, 9)])
def test_absdiff_numerators(ctx, w, h, b):
    img = _weights_image(w, h, 0)
    num, den, info = _sums(ctx, "tc", img, b, 0.0, "Abs. diff. of StdDevs")
    _, a = _expected_a(img, b, info)
    a = a.astype(np.float64)
    d = np.abs(a[:, None] - a[None])
    wt = np.exp2(-d * d)
    ws = np.sqrt(1.4426950408889634 / np.float64(np.float32(np.float32(info.noise_var) + np.float32(1e-7))))
    np.testing.assert_allclose(den, wt.sum(1), rtol=1e-6)
    # within a slice ex2.approx (2^-22) and FP32 sums of 32
    np.testing.assert_allclose(num, (d * wt).sum(1) / ws, rtol=2e-6)


# Contrast from all slabs factorised to slabs whose every weight underflows; both bars as in
# the parity tests (1e-5 of FP64, or 1.25 times the FP32 reference's own deviation).
@pytest.mark.parametrize("metric", ["Pearson's R", "SSIM", "NRMSE"])
@pytest.mark.parametrize("amp", [(5.0, 20.0), (50.0, 200.0), (500.0, 60000.0)])
def test_pair_forms_against_fp64(ctx, metric, amp):
    img = synth.normalize_input(synth.spot_image(101, 83, 6, seed=11, amp_range=amp))
    ctx.set_engine("tc")
    for c in (0.0, 1.0):
        out, _ = clutils.global_map_host(metric, img, 5, 5, c, ctx=ctx)
        j = oracle.global_map(metric, img, 5, 5, c, precision="f64")["map"]
        r = oracle.global_map(metric, img, 5, 5, c)["map"]
        assert float(np.max(np.abs(out - j))) <= max(1e-5, 1.25 * float(np.max(np.abs(r - j)))), (metric, amp, c)


@pytest.mark.parametrize("bw,bh", [(3, 3), (3, 7), (15, 15), (17, 17)])
@pytest.mark.parametrize("metric", ["Pearson's R", "NRMSE"])
def test_block_sizes(ctx, metric, bw, bh):
    """Every block size runs on the tensor cores, 17x17 and NRMSE of large blocks too."""
    img = synth.normalize_input(synth.spot_image(58, 52, 4, seed=bw))
    ctx.set_engine("tc")
    out, info = clutils.global_map_host(metric, img, bw, bh, 0.0, ctx=ctx)
    assert info["engine"] == _lib.ENGINE_TC
    j = oracle.global_map(metric, img, bw, bh, 0.0, precision="f64")["map"]
    assert float(np.max(np.abs(out - j))) <= 1e-5


# K at the edges of the operand's blocks of 16 (no tail, one element, fifteen) and of the two
# launch shapes (one CTA per tile, a pair, chunked stages); ragged n.
@pytest.mark.parametrize("k", [1, 15, 16, 17, 31, 32, 33, 48, 64, 100, 119, 144, 161, 192])
@pytest.mark.parametrize("n", [1, 129, 700])
def test_split_operand_rowdot(ctx, k, n):
    rng = np.random.default_rng(1000 * k + n)
    u = rng.normal(size=(n, k)).astype(np.float32)
    u /= np.linalg.norm(u, axis=1, keepdims=True).astype(np.float32)
    w1 = rng.uniform(-1, 1, n).astype(np.float32)
    num, den = np.zeros(n), np.zeros(n)
    ctx.check(ctx._L.sred_debug_gram_rowdot(ctx.h, _lib.ENGINE_TC, u, w1, np.abs(w1), n, k, num, den), "rowdot")
    U, w = u.astype(np.float64), w1.astype(np.float64)
    G = U @ U.T
    # per pair: 3 2^-22 |u_p||u_q| left out of the split and 2^-22 from the accumulation, and the
    # subnormal step of the unscaled mid parts, 2^-25 sqrt(K) each way; FP32 row and column sums
    err = 4 * 2.0 ** -22 + 2.0 ** -24 * np.sqrt(k)
    bound = np.abs(w) * (err * np.abs(w).sum() + 2e-6 * (np.abs(G) @ np.abs(w)))
    assert np.all(np.abs(num - w * (G @ w)) <= bound + 1e-30)
    np.testing.assert_allclose(den, n * np.abs(w) + np.abs(w).sum(), rtol=1e-6)
