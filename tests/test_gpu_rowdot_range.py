"""The engines' row products of vectors far from unit length: FP16 parts end at 65504 and
thin out below 2^-14, which the diagnostics' scaling keeps away from."""
import numpy as np
import pytest

from sred_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-9, 1e-4, 1.0, 1e5, 3e8])
@pytest.mark.parametrize("k", [5, 21, 49, 150])
@pytest.mark.parametrize("engine", [_lib.ENGINE_TC, _lib.ENGINE_FP32])
def test_scaled_vectors(engine, k, scale):
    ctx = _lib.Context(0, "tc")
    n = 300
    rng = np.random.default_rng(k)
    u = (rng.normal(size=(n, k)) / np.sqrt(k) * scale).astype(np.float32)
    w1 = rng.uniform(-1, 1, n).astype(np.float32)
    w2 = np.zeros(n, np.float32)  # no self pair is set to 1
    num, den = np.zeros(n), np.zeros(n)
    ctx.check(ctx._L.sred_debug_gram_rowdot(ctx.h, engine, u, w1, w2, n, k, num, den), "rowdot")
    U, w = u.astype(np.float64), w1.astype(np.float64)
    # per pair 3 2^-22 |u_p||u_q| of the split and (steps + 1) 2^-23 of the accumulation (an MMA of
    # 16 a step), and the FP32 row sums
    steps = 3 * k / 16 + 3 if engine == _lib.ENGINE_TC else k
    length = np.linalg.norm(U, axis=1)
    bound = np.abs(w) * length * (3 * 2.0 ** -22 + (steps + 1) * 2.0 ** -23) * (length @ np.abs(w))
    bound += np.abs(w) * 2e-6 * (np.abs(U @ U.T) @ np.abs(w))
    assert np.all(np.abs(num - w * (U @ (U.T @ w))) <= bound)
    assert np.all(den == 0)
