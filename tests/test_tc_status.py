"""A failed alignment check of the tensor-core kernel is not reported as a wait that ran out
(common.cuh, tc_status_error, compiled for the host). No GPU is used."""
import shutil
import subprocess
from pathlib import Path

import pytest

from sred_b200 import _lib

HERE = Path(__file__).resolve().parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def test_status_words(tmp_path):
    if not Path(NVCC).exists():
        pytest.skip("nvcc not available")
    out = tmp_path / "tc_status_check"
    cmd = [NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{HERE.parent / 'include'}",
           str(HERE / "native" / "tc_status_check.cu"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [line.split(" ", 2) for line in subprocess.check_output([str(out)], text=True).splitlines()]
    assert [int(s) for s, _, _ in lines] == [1, 2, 3, 4, 5]
    for s, e, msg in lines:
        if int(s) == 5:  # the kernel's own name for it: ST_ALIGNMENT = kTcUnaligned
            assert int(e) == _lib.ERR_LAUNCH and "aligned" in msg
        else:
            assert int(e) == _lib.ERR_TIMEOUT and "wait" in msg
