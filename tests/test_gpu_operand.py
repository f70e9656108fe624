"""Numerators and denominators of small-block maps on the tensor cores against 64 bits: the
spread of their quotient, which the normalisation of a map does not take out (a common
factor, as the MMAs' truncation gives, it does)."""
import ctypes as C
import math

import numpy as np
import pytest

from sred_b200 import _lib, synth

pytestmark = pytest.mark.gpu


# Blocks of 5 (one operand tail), 7 and 13 (padded blocks), 21 (a block and a tail) pixels.
@pytest.mark.parametrize("bw,bh", [(3, 3), (3, 5), (5, 5), (3, 19)])
def test_quotient_spread_of_small_blocks(bw, bh):
    import torch
    ctx = _lib.Context(0, "tc")
    w, h = 110, 97
    img = synth.normalize_input(synth.spot_image(w, h, 8, seed=5, random_fraction=0.3))
    d = torch.from_numpy(img).cuda()
    part = torch.zeros(2 * w * h, dtype=torch.float64, device="cuda")
    info = _lib.RunInfo()
    ctx.check(ctx._L.sred_global_map_2d_shard_sums(ctx.h, b"Pearson's R", C.c_void_p(d.data_ptr()), w, h, bw, bh, 0.0, 0,
                                                   1, C.c_void_p(part.data_ptr()), 2 * w * h, None, C.byref(info)),
              "shard_sums")
    n = int(info.n_relevant - info.n_flat)
    got = part[:n] / part[n:2 * n]
    rw, rh = bw // 2, bh // 2
    offs = [(y, x) for y in range(-rh, rh + 1) for x in range(-rw, rw + 1)
            if np.float32(x * x) / np.float32(rw * rw) + np.float32(y * y) / np.float32(rh * rh) <= 1]
    x = torch.stack([d.double()[rh + dy:h - rh + dy, rw + dx:w - rw + dx].reshape(-1) for dy, dx in offs], 1)
    assert x.shape[0] == n  # relevance constant 0: every block, none flat
    u = x - x.mean(1, keepdim=True)
    norm = u.square().sum(1).sqrt()
    u /= norm[:, None]
    s = norm / math.sqrt(len(offs) - 1)
    c = math.sqrt(math.log2(math.e) / float(np.float32(np.float32(info.noise_var) + np.float32(1e-7))))
    wt = torch.exp2(-((s[:, None] - s[None]) * c).square())
    t = ((u @ u.T) / (1 + 1e-7 / (s[:, None] * s[None]))).clamp(min=0) * wt
    err = got / (t.sum(1) / wt.sum(1)) - 1
    # Elements of 24 bits leave the FP32 sums of the pair terms and the weights' 2^-22, averaged over
    # thousands of pairs: 1.2e-8 to 1.5e-8 at K = 5. Elements of 22 bits and a sign are off by up to
    # 2^-24 each (3.4e-8 root mean square at most, 2e-8 over a vector), which adds up to 2.5e-8.
    assert float(err.std()) < 2.0e-8
    assert float(err.abs().max()) < 5e-7
