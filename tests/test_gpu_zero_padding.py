"""Ragged arrays have blocks that hold padding only, all zero: they call for no zero rule, and
change nothing where a zero block of items calls for it.  Non-finite items in the last rows and
columns, next to the padding; whole-number operands make every other sum exact, so the result
equals the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

CASES = [
    # M, K, N, chunk and block extents along m, k, n
    (300, 257, 200, (128, 128, 128), (32, 32, 32)),      # the last chunks mostly padding
    (65, 65, 65, (64, 64, 64), (16, 16, 16)),            # one item beyond a whole chunk
    (50, 47, 31, (50, 47, 31), (32, 32, 16)),            # blocks beyond the chunk's edge
    (33, 40, 17, (32, 40, 16), (8, 8, 8)),
]


@pytest.mark.parametrize("zero", [False, True], ids=["padding", "zeroblock"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:3])))
def test_padding_blocks(ia, ctx, case, dtype, zero):
    M, K, N, (cm, ck, cn), (bm, bk, bn) = case
    rng = np.random.default_rng(M)
    A, B = rng.integers(-8, 9, (M, K)).astype(dtype), rng.integers(-8, 9, (K, N)).astype(dtype)
    x = rng.integers(-8, 9, K).astype(dtype)
    if zero:
        A[:bm, :bk] = 0
        x[:bk] = 0
    A[M - 1, K - 1], A[0, K - 1] = np.nan, np.inf
    B[K - 1, N - 1], B[0, 0] = -np.inf, np.nan
    dt = O.DTYPE_DOUBLE if dtype is np.float64 else O.DTYPE_FLOAT
    a = ia.Container.from_numpy(ctx, A, (cm, ck), (bm, bk))
    ga, ach = O.encode_array(A, (cm, ck), (bm, bk))
    for v, ch, bl in ((B, (ck, cn), (bk, bn)), (x, (ck,), (bk,))):
        b = ia.Container.from_numpy(ctx, v, ch, bl)
        gb, bch = O.encode_array(v, ch, bl)
        vec = v.ndim == 1
        out, ob = ((cm,), (bm,)) if vec else ((cm, cn), (bm, bn))
        gc = O.Geom((M,) if vec else (M, N), out, ob, A.itemsize)
        got = (ia.opt_gemv if vec else ia.opt_gemm)(ctx, a, b, out, ob).to_numpy()
        ref = (O.opt_gemv if vec else O.opt_gemm)(ga, ach, gb, bch, gc, dt)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        np.testing.assert_array_equal(got, ref)
        b.free()
    a.free()
