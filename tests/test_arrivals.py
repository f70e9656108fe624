"""Every arrival of the tensor-core kernel's epilogue that lets a copy overwrite a buffer of
shared memory follows a fence in the same block of statements, and the one that hands tensor
memory on follows tcgen05.fence::before_thread_sync. A race is not shown by running it; the
source is read instead."""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "sred_b200" / "csrc" / "global_tc.cu").read_text()


def _calls(name):
    body = SOURCE[SOURCE.index("k_gram_tc("):]
    at = [m.start() for m in re.finditer(name + r"\(", body)]
    assert at, name
    return [(body[:i], body[body.rindex("{", 0, i):i], body[i:i + 60]) for i in at]


def test_arrivals_follow_a_fence():
    relaxed = re.findall(r"__device__ __forceinline__ void (\w+)\([^)]*\) \{[^}]*mbarrier\.arrive\.relaxed", SOURCE)
    assert len(relaxed) == SOURCE.count("mbarrier.arrive.relaxed")
    assert set(relaxed) == {"mbar_arrive_tmem", "mbar_arrive_fenced"}
    for _, block, call in _calls("mbar_arrive_fenced"):
        assert "fence_reads();" in block, call
    for before, _, call in _calls("mbar_arrive_tmem"):
        tail = before[before.rindex("tc_fence_before();"):]
        assert "tmem_" not in tail and "tile_" not in tail, call  # nothing reads tensor memory in between
