"""The default chunk of a time-lapse: an eighth of the stack in 2 to 32 MiB, and 32 MiB where
the output is pageable, whose downloads overlap nothing (compiled for the host). No GPU is used."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    if not Path(NVCC).exists():
        pytest.skip("nvcc not available")
    out = tmp_path_factory.mktemp("chunk") / "stack_chunk_check"
    cmd = [NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{HERE.parent / 'include'}",
           str(HERE / "native" / "stack_chunk_check.cu"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return lambda *a: int(subprocess.check_output([str(out), *map(str, a)], text=True))


@pytest.mark.parametrize("frames,plane,pinned,pageable", [(24, 512 * 512, 3, 32), (100, 256 * 256, 12, 128),
                                                          (2000, 512 * 512, 32, 32), (1, 64, 8192, 131072),
                                                          (3, 4096 * 4096, 0, 0)])
def test_default_chunk(chunk, frames, plane, pinned, pageable):
    assert chunk(frames, plane, 0) == pinned
    assert chunk(frames, plane, 1) == pageable
