"""Global maps of different block sizes from several threads, a context each: the kernels'
shared memory differs by block size, and no launch may meet another thread's limit."""
import threading

import numpy as np
import pytest

from sred_b200 import _lib, clutils, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["tc", "fp32"])
def test_block_sizes_from_several_threads(engine):
    img = synth.normalize_input(synth.spot_image(62, 54, 4, seed=3))
    sizes = [3, 7, 11, 15]
    alone = {}
    for b in sizes:
        alone[b], _ = clutils.global_map_host("Pearson's R", img, b, b, 0.0, ctx=_lib.Context(0, engine))
    failed = []

    def work(b):
        try:
            ctx = _lib.Context(0, engine)
            for _ in range(100):
                out, _ = clutils.global_map_host("Pearson's R", img, b, b, 0.0, ctx=ctx)
                # (FP64 atomic sums in another order: an FP32 rounding at most)
                if float(np.abs(out - alone[b]).max()) > 2.0 ** -23:
                    failed.append((b, "differs"))
        except Exception as e:  # noqa: BLE001 (reported below)
            failed.append((b, str(e)))

    threads = [threading.Thread(target=work, args=(b,)) for b in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == []
