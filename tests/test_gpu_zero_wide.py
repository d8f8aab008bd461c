"""The non-finite scan of the block-pair products at the edges of its 1024-item row pieces: NaN and
infinities in the pieces' first and last columns and the array's last row, some facing zero blocks.
Whole-number operands make every sum exact, so the result equals the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 1023, 1024, 1025, 2049])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_row_pieces(ia, ctx, K, dtype):
    rng = np.random.default_rng(K)
    M, N, ch, bl = 21, 1030, (16, 512), (8, 64)
    A, B = rng.integers(-8, 9, (M, K)).astype(dtype), rng.integers(-8, 9, (K, N)).astype(dtype)
    chb = (512, 16), (64, 8)
    A[:8, :64] = 0                                       # zero blocks on both sides
    B[-(K % 64 or 64):, :8] = 0
    for c in {0, 1022, 1023, 1024, K - 1} & set(range(K)):
        A[M - 1 - c % 2, c] = np.nan
        B[c, 5] = np.inf
    for c in (0, 1023, 1024, N - 1):
        B[K - 1, c] = np.nan
    a = ia.Container.from_numpy(ctx, A, ch, bl)
    b = ia.Container.from_numpy(ctx, B, *chb)
    got = ia.opt_gemm(ctx, a, b, (16, 16), (8, 8)).to_numpy()
    ga, ach = O.encode_array(A, ch, bl)
    gb, bch = O.encode_array(B, *chb)
    dt = O.DTYPE_DOUBLE if dtype is np.float64 else O.DTYPE_FLOAT
    ref = O.opt_gemm(ga, ach, gb, bch, O.Geom((M, N), (16, 16), (8, 8), A.itemsize), dt)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(got, ref)
    a.free()
    b.free()
