"""Block maps of tall and of wide blocks on images of several hundred tiles, bit for bit:
blocks whose four-column tile fits twice into an SM (3x81), once (3x101) and not at
all (3x195 and taller), up to the tallest block there is (3x509); rows of one
element, runs of equal rows, rows of every remainder of four. Through the context and through the
allocation-free entry point, which takes a block by the tile of 48 KB it documents."""
import ctypes as C

import numpy as np
import pytest

from sred_b200 import _lib, clutils
from test_gpu_block_map import _expected, _offsets, _reference

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return _lib.Context(0, "tc")


@pytest.mark.parametrize("w,h,bw,bh,metric", [
    (1024, 480, 3, 81, "Pearson's R"), (1024, 480, 3, 101, "Pearson's R"), (1024, 480, 3, 195, "Pearson's R"),
    (1030, 481, 3, 201, "SSIM"), (1024, 480, 3, 321, "NRMSE (inverted)"), (1024, 530, 3, 509, "Abs. Diff. of StdDevs."),
    (1021, 480, 5, 101, "Pearson's R"), (1024, 480, 7, 71, "SSIM"), (1024, 480, 101, 3, "Pearson's R"),
    (1024, 480, 401, 3, "NRMSE (inverted)"), (1024, 480, 25, 25, "SSIM"), (60, 480, 3, 321, "SSIM")])
def test_tall_and_wide_blocks(ctx, w, h, bw, bh, metric):
    import torch
    rng = np.random.default_rng(bw * bh)
    img = (rng.random((h, w), dtype=np.float32) * np.float32(100)).astype(np.float32)
    offs = _offsets(bw, bh)
    ref = _reference(img, offs, bw, bh, h // 2, w // 2)
    exp = _expected(metric, img, ref, offs, bw // 2, bh // 2, True)
    d_in = torch.from_numpy(img).cuda()
    d_out = torch.empty_like(d_in)
    clutils.block_map_device(metric, d_in.data_ptr(), w, h, 1, ref, 0.0, True, d_out.data_ptr(), ctx=ctx)
    assert np.array_equal(d_out.cpu().numpy(), exp)
    if 4 * (32 + 2 * (bw // 2)) * (16 + 2 * (bh // 2)) + 8 * len(offs) <= 48 * 1024:
        d_out.zero_()
        px = np.ascontiguousarray(ref.pixels, np.float32)
        status = ctx._L.sred_block_map_2d_device_noalloc(metric.encode(), C.c_void_p(d_in.data_ptr()), w, h, 1, px, px.size, bw,
                                                    bh, float(ref.mean), float(ref.std), 1, C.c_void_p(d_out.data_ptr()),
                                                    None)
        assert status == _lib.OK
        assert np.array_equal(d_out.cpu().numpy(), exp)


def test_block_sizes_from_several_threads():
    """Launches of different tile sizes from threads with a context each."""
    import threading
    import torch
    rng = np.random.default_rng(0)
    img = rng.random((420, 64), dtype=np.float32)
    d_in = torch.from_numpy(img).cuda()
    failed = []

    def work(bw, bh):
        try:
            c = _lib.Context(0, "tc")
            offs = _offsets(bw, bh)
            ref = _reference(img, offs, bw, bh, 210, 32)
            out = torch.empty_like(d_in)
            torch.cuda.synchronize()
            for _ in range(200):
                clutils.block_map_device("Pearson's R", d_in.data_ptr(), 64, 420, 1, ref, 0.0, True, out.data_ptr(), ctx=c)
            if not np.array_equal(out.cpu().numpy(), _expected("Pearson's R", img, ref, offs, bw // 2, bh // 2, True)):
                failed.append((bw, bh))
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append((bw, bh, str(e)))

    # tiles of 55, 83 and 111 KB
    threads = [threading.Thread(target=work, args=s) for s in ((3, 191), (3, 291), (3, 391), (3, 191))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == []
