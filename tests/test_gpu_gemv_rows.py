"""The row-per-warp GEMV at the edges of its groups of 8 loads per lane: 16-byte loads of 32 lanes,
rows of whole groups, one item more and less, rows shorter than a load.  Blocks of odd width (and a
transposed view) keep the call off the decode-fused kernel; whole numbers make every sum exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loads", [0, 1, 224, 225, 256, 257, 512])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("tail", [0, 1, -1])
def test_row_groups(ia, ctx, dtype, loads, tail):
    K = max(loads * (16 // np.dtype(dtype).itemsize) + tail, 1)
    rng = np.random.default_rng(K)
    A, x = rng.integers(-8, 9, (37, K)).astype(dtype), rng.integers(-8, 9, K).astype(dtype)
    ref = A.astype(np.float64) @ x.astype(np.float64)
    b = min(K, 51)
    v = ia.Container.from_numpy(ctx, x, (K,), (b,))
    a = ia.Container.from_numpy(ctx, A, (20, K), (10, b))
    t = ia.Container.from_numpy(ctx, np.ascontiguousarray(A.T), (K, 20), (b, 10))
    for m in (a, t.transpose()):
        got = ia.matmul(ctx, m, v, (20,), (10,)).to_numpy()
        np.testing.assert_array_equal(got.astype(np.float64), ref)
    for c in (a, t, v):
        c.free()
