"""The tensor-core engine's ring of operand stages: the stage that the epilogue releases
for a tile is the one its last operands lie in, for every block size and launch shape
(compiled for the host from the library's own source), and maps whose tiles take more
stages than the ring has, with enough tiles for it to wrap."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_released_stage_of_every_shape(tmp_path):
    if not Path(NVCC).exists():
        pytest.skip("nvcc not available")
    out = tmp_path / "ring_stage_check"
    cmd = [NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
           f"-I{HERE.parent / 'include'}", str(HERE / "native" / "ring_stage_check.cu"), "-o", str(out), "-lcuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    shapes = [tuple(map(int, line.split())) for line in subprocess.check_output([str(out)], text=True).splitlines()]
    assert {k for k, *_ in shapes} >= set(range(1, 213))
    assert any(nst > ring for _, _, _, nst, ring, _ in shapes)
    assert [s for s in shapes if s[-1] >= 0] == []


# K = 175, 197 and 185: seven stages a tile in a ring of five; 8,448 blocks and more are 34 column
# tiles, several tiles for every pair of CTAs.
@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["Pearson's R", "SSIM", "NRMSE"])
@pytest.mark.parametrize("w,h,bw,bh", [(110, 112, 15, 17), (112, 104, 17, 17), (111, 110, 13, 21)])
def test_maps_of_wrapping_rings(metric, w, h, bw, bh):
    import oracle
    from sred_b200 import _lib, clutils, synth
    ctx = _lib.Context(0, "tc")
    img = synth.normalize_input(synth.spot_image(w, h, 8, seed=bw + bh))
    out, info = clutils.global_map_host(metric, img, bw, bh, 0.0, ctx=ctx)
    assert info["engine"] == _lib.ENGINE_TC and info["n_relevant"] >= 8000
    j = oracle.global_map(metric, img, bw, bh, 0.0, precision="f64")["map"]
    # the bar of the parity tests
    assert float(np.max(np.abs(out - j))) <= 1e-5
