"""What SSIM's factorised slabs neglect is bounded (global_tc.cu, ssim_split_bounded, compiled
for the host): 2^-21 for the weight without its first-order term or (6.9e-4)^2 / 2 with it, and
2^-22 for the curvature of 1/(sigma_p^2 + sigma_q^2 + c2); weighted NRMSE's row factors are
normal numbers (row_factors_normal). No GPU is used."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_neglected_terms(tmp_path):
    if not Path(NVCC).exists():
        pytest.skip("nvcc not available")
    out = tmp_path / "ssim_slab_check"
    cmd = [NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
           f"-I{HERE.parent / 'include'}", str(HERE / "native" / "ssim_slab_check.cu"), "-o", str(out), "-lcuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    tried, accepted, wide, worst = subprocess.check_output([str(out)], text=True).split()
    assert int(accepted) > int(tried) // 10 and int(wide) > 1000
    assert float(worst) <= 2.0 ** -21 + 2.0 ** -22 + 5e-8  # (1e-8 and less of FP32 rounding in the bound)
