"""Timed workloads of the repetition maps: what they are, how a program calls
them, what they have to move and compute, and their values in 64 bits.

Four paths, through the functions a program calls (``sred_b200.clutils``): the
2D and 3D global maps (every relevant block against every other one) and the
2D and 3D block maps (one reference block against every block). Images are
synthetic spot images with shot and read noise, min-max normalised as the
commands do it (``sred_b200.synth``). A program keeps one library context per
engine for all its images, so the contexts are made once per process.
"""
import ctypes
import math

import numpy as np
import torch

from sred_b200 import _lib, clutils, synth, utils

PEARSON, SSIM = "Pearson's R", "SSIM"
NRMSE, ABSDIFF = "NRMSE", "Abs. diff. of StdDevs"  # global maps
NRMSE_B, ABSDIFF_B = "NRMSE (inverted)", "Abs. Diff. of StdDevs."  # block maps

# Share of the interior blocks with sigma^2 >= the noise variance in these images
# (relevance constant 1), for the work estimate.
RELEVANT_SHARE = {2: 0.73, 3: 0.35}


def _g2(name, metric, w, h, bw, bh, relevance, engine="tc", io="device"):
    return {"name": name, "path": "global2d", "metric": metric, "w": w, "h": h, "bw": bw, "bh": bh,
            "relevance": relevance, "engine": engine, "io": io}


def _g3(name, metric, w, h, d, bw, bh, bd, relevance):
    return {"name": name, "path": "global3d", "metric": metric, "w": w, "h": h, "d": d, "bw": bw, "bh": bh, "bd": bd,
            "relevance": relevance, "engine": "tc", "io": "device"}


def _b2(name, metric, w, h, frames, bw, bh, relevance, io="device"):
    return {"name": name, "path": "block2d", "metric": metric, "w": w, "h": h, "frames": frames, "bw": bw, "bh": bh,
            "relevance": relevance, "engine": "tc", "io": io}


def _b3(name, metric, w, h, d, bw, bh, bd, relevance):
    return {"name": name, "path": "block3d", "metric": metric, "w": w, "h": h, "d": d, "bw": bw, "bh": bh, "bd": bd,
            "relevance": relevance, "engine": "tc", "io": "device"}


def listed():
    return [
        # The dialog's defaults (5x5, Pearson, relevance 0) on a small field of view.
        _g2("global 256 5x5 pearson", PEARSON, 256, 256, 5, 5, 0.0),
        # A camera frame with 9x9 blocks and the relevance mask: the benchmark's map.
        _g2("global 1024 9x9 pearson", PEARSON, 1024, 1024, 9, 9, 1.0),
        # Structural similarity of a mid-size crop, from and to host memory as the command runs it.
        _g2("global 512 9x9 ssim host", SSIM, 512, 512, 9, 9, 1.0, io="host"),
        # A ragged crop, anisotropic blocks, every metric's general case.
        _g2("global 611x433 11x7 nrmse", NRMSE, 611, 433, 11, 7, 0.5),
        # Large structures: the largest block of the benchmark's batch.
        _g2("global 640x576 15x15 pearson", PEARSON, 640, 576, 15, 15, 1.0),
        # The metric without block dot products.
        _g2("global 500x381 7x7 absdiff", ABSDIFF, 500, 381, 7, 7, 1.0),
        # The engine of a context made without naming one (plain FP32), a small host image.
        _g2("global 233x180 5x5 fp32 host", PEARSON, 233, 180, 5, 5, 1.0, engine="fp32", io="host"),
        # A volume with the 3D blocks of the benchmark.
        _g3("global3d 128x128x48 5x5x5", PEARSON, 128, 128, 48, 5, 5, 5, 1.0),
        # One reference block over a time-lapse that is on the GPU.
        _b2("block 1024 x16 15x15 pearson", PEARSON, 1024, 1024, 16, 15, 15, 0.0),
        # The smallest call: one host image, one reference block, with the relevance mask.
        _b2("block 256 9x9 ssim host", SSIM, 256, 256, 1, 9, 9, 1.0, io="host"),
        # A host time-lapse streamed through the GPU.
        _b2("stack 512 x24 11x11 nrmse", NRMSE_B, 512, 512, 24, 11, 11, 0.0, io="host"),
        # One reference block over a volume.
        _b3("block3d 256x256x64 5x5x5", PEARSON, 256, 256, 64, 5, 5, 5, 0.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: image sides over their logarithm, odd
    sizes and anisotropic blocks among them, every metric and relevance constant."""
    path = rng.choices(["global2d", "global3d", "block2d", "block3d"], [5, 2, 3, 2])[0]
    rel = rng.choice([0.0, 0.5, 1.0, 1.5])
    if path == "global2d":
        engine = rng.choices(["tc", "fp32"], [4, 1])[0]
        bw, bh = rng.choice([3, 5, 7, 9, 11, 13, 15]), rng.choice([3, 5, 7, 9, 11, 13, 15])
        if rng.random() < 0.6:
            bh = bw
        lim = 560 if engine == "tc" else 300
        w, h = _log(rng, 72, lim), _log(rng, 72, lim)
        c = _g2("", rng.choice([PEARSON, PEARSON, SSIM, NRMSE, ABSDIFF]), w, h, bw, bh, rel, engine,
                rng.choice(["device", "host"]))
    elif path == "global3d":
        bw, bd = rng.choice([3, 5, 7]), rng.choice([3, 5])
        c = _g3("", rng.choice([PEARSON, SSIM, NRMSE, ABSDIFF]), _log(rng, 32, 110), _log(rng, 32, 110),
                _log(rng, 12, 36), bw, bw, bd, rel)
    elif path == "block2d":
        bw, bh = rng.choice([3, 5, 7, 9, 11, 13, 15, 19]), rng.choice([3, 5, 7, 9, 11, 13, 15, 19])
        io = rng.choice(["device", "host"])
        w, h = _log(rng, 96, 1100), _log(rng, 96, 1100)
        frames = max(1, min(_log(rng, 1, 24), (8 << 20) // (w * h)))
        c = _b2("", rng.choice([PEARSON, SSIM, NRMSE_B, ABSDIFF_B]), w, h, frames, bw, bh, rel, io)
    else:
        bw, bh, bd = rng.choice([3, 5, 7]), rng.choice([3, 5, 7]), rng.choice([3, 5])
        c = _b3("", rng.choice([PEARSON, SSIM, NRMSE_B, ABSDIFF_B]), _log(rng, 48, 256), _log(rng, 48, 256),
                _log(rng, 16, 48), bw, bh, bd, rel)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# What a program has in hand, and its call
# ---------------------------------------------------------------------------

_contexts = {}


def _context(engine):
    if engine not in _contexts:
        _contexts[engine] = clutils.get_open_cl_resources(engine=engine)
    return _contexts[engine]


def _lattice(w, h):
    return max(2, int(round(math.sqrt(w * h) / 12.8)))


def _image(case, seed):
    """float32 [h, w] (frames: [f, h, w]) or [d, h, w], min-max normalised."""
    if "d" in case:
        v = synth.spot_volume(case["w"], case["h"], case["d"], max(2, _lattice(case["w"], case["h"])),
                              max(1, case["d"] // 8), seed=seed)
        return synth.normalize_input(v)
    img = synth.spot_image(case["w"], case["h"], _lattice(case["w"], case["h"]), seed=seed, random_fraction=0.3)
    f = case.get("frames", 1)
    if f == 1:
        return synth.normalize_input(img)
    # a time-lapse: the same field, fading, with new read noise in every frame
    rng = np.random.default_rng(seed + 1)
    out = np.empty((f, case["h"], case["w"]), np.float32)
    for i in range(f):
        noise = rng.standard_normal(img.shape, dtype=np.float32)
        out[i] = synth.normalize_input(img * np.float32(1.0 - 0.01 * i) + np.float32(5.0) * noise)
    return out


def _reference_block(case, img):
    """The block at a third of the image (of the first frame, or of the volume)."""
    if case["path"] == "block3d":
        z, y, x = case["d"] // 3, case["h"] // 3, case["w"] // 3
        return utils.get_reference_block_3d(img[z:z + case["bd"], y:y + case["bh"], x:x + case["bw"]])
    a = img if img.ndim == 2 else img[0]
    y, x = case["h"] // 3, case["w"] // 3
    return utils.get_reference_block_2d(a[y:y + case["bh"], x:x + case["bw"]])


def _pinned(shape):
    """Page-locked host memory, as a program that streams frames keeps it."""
    return torch.empty(shape, dtype=torch.float32, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    img = _image(case, seed)
    s = {"case": case, "ctx": _context(case["engine"])}
    if case["path"].startswith("block"):
        s["block"] = _reference_block(case, img)
    if case["io"] == "device":
        s["img"] = torch.from_numpy(img).cuda()
        s["out"] = torch.empty_like(s["img"])
        torch.cuda.synchronize()
    else:
        s["img"], s["out"] = _pinned(img.shape), _pinned(img.shape)
        s["img"][...] = img
    return s


def run(s):
    c, ctx = s["case"], s["ctx"]
    args = (c["metric"],)
    if c["io"] == "device":
        p_in, p_out = s["img"].data_ptr(), s["out"].data_ptr()
        if c["path"] == "global2d":
            clutils.global_map_device(*args, p_in, c["w"], c["h"], c["bw"], c["bh"], c["relevance"], True, p_out,
                                      ctx=ctx)
        elif c["path"] == "global3d":
            clutils.global_map_3d_device(*args, p_in, c["w"], c["h"], c["d"], c["bw"], c["bh"], c["bd"],
                                         c["relevance"], True, p_out, ctx=ctx)
        elif c["path"] == "block2d":
            clutils.block_map_device(*args, p_in, c["w"], c["h"], c["frames"], s["block"], c["relevance"], True,
                                     p_out, ctx=ctx)
        else:
            clutils.block_map_3d_device(*args, p_in, c["w"], c["h"], c["d"], s["block"], c["relevance"], True, p_out,
                                        ctx=ctx)
        return s["out"]
    if c["path"] == "global2d":
        out, _ = clutils.global_map_host(*args, s["img"], c["bw"], c["bh"], c["relevance"], True, out=s["out"],
                                         ctx=ctx)
        return out
    if c["frames"] == 1:
        img = utils.InputImage2D(s["img"].reshape(-1), c["w"], c["h"])
        return clutils.calculate_block_repetition_map_2d(*args, img, s["block"], c["relevance"], True, ctx=ctx)
    return clutils.block_map_stack(*args, s["img"], s["block"], c["relevance"], True, out=s["out"], ctx=ctx)


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------

def _offsets(case):
    """The ellipse's (ellipsoid's) offsets in raster order, FP32 arithmetic as the
    reference has it (java/GlobalRepetition2D_.java:102-111, java/Utils.java:1075-1085)."""
    f = np.float32
    r = [case["bd"] // 2] if "bd" in case else []
    r += [case["bh"] // 2, case["bw"] // 2]
    out = []
    for o in np.ndindex(*[2 * k + 1 for k in r]):
        d = [a - k for a, k in zip(o, r)]
        t = f(0)
        for v, k in zip(d[::-1], r[::-1]):  # x, then y, then z
            t = f(t + f(f(v) * f(v)) / f(k * k))
        if t <= f(1):
            out.append(tuple(d))
    return out


def work(case):
    """Bytes: the image once in, the map once out. Flops: the block statistics
    (4 K per block) and, where the metric correlates blocks, 2 K per pair: each
    unordered pair once in a global map, each block once in a block map."""
    k = len(_offsets(case))
    px = case["w"] * case["h"] * case.get("d", 1) * case.get("frames", 1)
    inner = (case["w"] - case["bw"] + 1) * (case["h"] - case["bh"] + 1)
    if "bd" in case:
        inner *= case["d"] - case["bd"] + 1
    inner *= case.get("frames", 1)
    flops = 4.0 * k * inner
    if case["metric"] not in (ABSDIFF, ABSDIFF_B):
        if case["path"].startswith("global"):
            n = inner * (1.0 if case["relevance"] == 0 else RELEVANT_SHARE[3 if "bd" in case else 2])
            flops += n * (n + 1) / 2 * 2 * k
        else:
            flops += 2.0 * k * inner
    return {"bytes": 8.0 * px, "flops": flops}


# ---------------------------------------------------------------------------
# The maps in 64 bits, with plain torch: every decision (which blocks are
# relevant, the noise variance) in FP32 in the reference's order, as the maps
# define it; every value in FP64.
# ---------------------------------------------------------------------------

EPS, C1, C2 = np.float32(1e-7), np.float32(0.0001), np.float32(0.0009)


def _views(a, offs, radii):
    """The interior shifted by each offset, one view per ellipse element."""
    for o in offs:
        yield a[tuple(slice(r + d, n - r + d) for r, d, n in zip(radii, o, a.shape))]


def _stats32(a, offs, radii):
    """FP32 local means and stds of the interior, the reference's order."""
    k = len(offs)
    s = None
    for v in _views(a, offs, radii):
        s = v.clone() if s is None else s + v
    mean = s / float(k)
    var = torch.zeros_like(mean)
    for v in _views(a, offs, radii):
        d = v - mean
        var = var + d * d
    return mean, torch.sqrt(var / float(k - 1))


def _noise_var_2d(a):
    """java/Utils.java:790-837 in FP32: the mean of the lowest 3% of the tile variances."""
    f = np.float32
    h, w = a.shape
    t = 8 if w * h <= 352 * 288 else 16
    tiles = a[:h // t * t, :w // t * t].reshape(h // t, t, w // t, t)
    m = torch.zeros(h // t, w // t, dtype=torch.float32, device=a.device)
    q = torch.zeros_like(m)
    for y in range(t):
        for x in range(t):
            v = tiles[:, y, :, x]
            m = m + v
            q = q + v * v
    m = m / float(t * t)
    var = np.sort((q / float(t * t) - m * m).cpu().numpy().ravel())
    n = int(f(f(0.03) * f(var.size)) + f(1))
    v = f(0)
    for x in var[:n]:
        v = f(v + x)
    v = f(abs(f(v / f(n))))
    return f(f(f(1) + f(f(0.001) * f(v - f(40)))) * v)


def _noise_var_3d(std):
    """java/Utils.java:1463-1498: the mean local variance, an FP32 raster-order sum."""
    s2 = (std * std).cpu().numpy().ravel()
    return np.float32(np.add.accumulate(s2, dtype=np.float32)[-1] / np.float32(min(s2.size, 1 << 24)))


def _normalised(m, sel):
    v = m[sel]
    if v.numel() == 0:
        return m
    lo, hi = v.min(), v.max()
    return torch.where(sel, (m - lo) / (hi - lo + float(EPS)), m)


def _placed(inner, like, radii):
    out = torch.zeros(like.shape, dtype=torch.float64, device=like.device)
    out[tuple(slice(r, n - r) for r, n in zip(radii, like.shape))] = inner
    return out


def _exact_global(case, a, offs, radii):
    vol = "bd" in case
    metric, k = case["metric"], len(offs)
    _, s32 = _stats32(a, offs, radii)
    nv = _noise_var_3d(s32) if vol else _noise_var_2d(a)
    thr = np.float32(nv * np.float32(case["relevance"]))
    s2 = s32 * s32
    mask, use = ~(s2 <= float(thr)), ~(s2 < float(thr))
    if bool((use & (s32 == 0)).any()):
        return None  # exactly flat blocks: none in these images
    x = torch.stack([v[use] for v in _views(a.double(), offs, radii)], 1)
    mu = x.mean(1)
    u = x - mu[:, None]
    del x
    nrm = u.square().sum(1).sqrt()
    sig = nrm / math.sqrt(k - 1)
    u /= nrm[:, None]
    n = sig.numel()
    ca = math.sqrt(math.log2(math.e) / float(np.float32(nv + EPS)))
    eps, c1, c2 = float(EPS), float(C1), float(C2)
    num = torch.zeros(n, dtype=torch.float64, device=a.device)
    den = torch.zeros_like(num)
    step = max(64, min(4096, int(6e9 / 8 / n)))
    for i in range(0, n, step):  # rows [i, j) against columns [i, n): the later rows get their terms from here
        j = min(n, i + step)
        sp, sq = sig[i:j, None], sig[None, i:]
        w = (sp - sq).mul_(ca).square_().neg_().exp2_()
        if metric == ABSDIFF:
            t = (sp - sq).abs_().mul_(w)
        else:
            t = u[i:j] @ u[i:].T
            if metric == PEARSON:
                t.div_(1.0 + eps / sp / sq).clamp_(min=0).mul_(w)
            elif metric == SSIM:
                t.mul_(sp).mul_(sq).mul_(2.0).add_(c2)
                t.div_((sp * sp + c2) + sq * sq)
                m = mu[i:j, None] * mu[None, i:]
                t.mul_((2.0 * m + c1).div_(m.square_().add_(c1))).mul_(w).clamp_(min=0)
                del m
            else:
                t.neg_().add_(1.0).mul_(sp).mul_(sq).mul_(2.0).add_((sp - sq).square_()).mul_((k - 1) / k)
                t.clamp_(min=0).sqrt_()
                if vol:
                    t.mul_(w)
        num[i:j] += t.sum(1)
        den[i:j] += w.sum(1)
        num[j:] += t[:, j - i:].sum(0)
        den[j:] += w[:, j - i:].sum(0)
        del t, w
    npx = float(min(int(mask.sum()), 1 << 24))
    m = torch.zeros(mask.shape, dtype=torch.float64, device=a.device)
    m[use] = num / (den * npx + eps)
    if metric in (NRMSE, ABSDIFF):
        m = torch.where(mask, torch.where(m == 0, torch.ones_like(m), 1.0 / m), m)
    if case["relevance"] > 0:
        m = m * mask
    return _placed(_normalised(m, mask), a, radii)


def _exact_block(case, a, offs, radii, ref):
    vol = "bd" in case
    metric, k = case["metric"], len(offs)
    _, s32 = _stats32(a, offs, radii)
    nv = (_noise_var_3d(s32) if vol else _noise_var_2d(a)) if case["relevance"] > 0 else np.float32(0)
    mask = ~(s32 * s32 <= float(np.float32(nv * np.float32(case["relevance"]))))
    if case["relevance"] == 0:
        mask = torch.ones_like(mask)
    d = a.double()
    px = [float(v) for v in ref.pixels]
    rm, rs = float(ref.mean), float(ref.std)
    mean = sum(_views(d, offs, radii)) / k
    std = (sum((v - mean).square() for v in _views(d, offs, radii)) / (k - 1)).sqrt()
    eps, c1, c2 = float(EPS), float(C1), float(C2)
    if metric == ABSDIFF_B:
        m = (rs - std).abs()
    elif metric == PEARSON and vol:
        # cl/kernelGetBlockPearson3D.cl: min-max, minus the block's mean, min-max again
        lo = torch.full_like(mean, math.inf)
        hi = -lo
        for v in _views(d, offs, radii):
            lo, hi = torch.minimum(lo, v), torch.maximum(hi, v)
        lo2 = 0.0 - mean  # the first normalisation's smallest value is 0
        hi2 = (hi - lo) / (hi - lo + eps) - mean
        cov = sum(p * (((v - lo) / (hi - lo + eps) - mean) - lo2) / (hi2 - lo2 + eps)
                  for p, v in zip(px, _views(d, offs, radii))) / (k - 1)
        m = (cov / (rs * std + eps)).clamp(min=0)
    else:
        cov = sum(p * (v - mean) for p, v in zip(px, _views(d, offs, radii))) / (k - 1)
        if metric == PEARSON:
            m = (cov / (rs * std + eps)).clamp(min=0)
        else:
            m = ((2 * rm * mean + c1) * (2 * cov + c2)
                 / ((rm * rm + mean * mean + c1) * (rs * rs + std * std + c2))).clamp(min=0)
    if metric == ABSDIFF_B:
        m = 1.0 - m if vol else 1.0 - (m - m.min()) / (m.max() - m.min() + eps)
    if case["relevance"] > 0:
        m = m * mask
    return _placed(_normalised(m, mask), a, radii)


def exact(case, seed):
    """None for the inverted NRMSE block map: it inverts a map normalised to
    start at 0, so its largest values are reciprocals of rounding differences."""
    if case["metric"] == NRMSE_B:
        return None
    img = _image(case, seed)
    a = torch.from_numpy(img).cuda()
    offs = _offsets(case)
    radii = ([case["bd"] // 2] if "bd" in case else []) + [case["bh"] // 2, case["bw"] // 2]
    if case["path"].startswith("global"):
        out = _exact_global(case, a, offs, radii)
    else:
        ref = _reference_block(case, img)
        if case["path"] == "block2d" and img.ndim == 3:
            out = torch.stack([_exact_block(case, f, offs, radii, ref) for f in a])
        else:
            out = _exact_block(case, a, offs, radii, ref)
    if out is None:
        return None
    return out if case["io"] == "device" else out.cpu().numpy().reshape(_shape(case))


def _shape(case):
    """Host calls: the one-image block map returns its pixels flat."""
    if case["path"] == "block2d" and case["frames"] == 1:
        return (case["w"] * case["h"],)
    return (case["frames"], case["h"], case["w"]) if case["path"] == "block2d" else (case["h"], case["w"])
