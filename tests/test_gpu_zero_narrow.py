"""The non-finite scan of the block-pair products on operands narrower than its 1024-item pieces,
which take several rows each: widths around the powers of two, last rows that fill a part of a piece.
Whole-number operands make every sum exact, so the result equals the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 8, 31, 33, 511, 512, 513])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rows_of_a_piece(ia, ctx, K, dtype):
    rng = np.random.default_rng(K)
    M, N = 1024 // K + 203, 37                           # a whole piece of rows and a part of one
    bl, ch, chb = (8, 16), (64, 48), (48, 16)
    A, B = rng.integers(-8, 9, (M, K)).astype(dtype), rng.integers(-8, 9, (K, N)).astype(dtype)
    A[16:24] = 0                                         # zero blocks, in both operands
    B[:16, 16:24] = 0
    for i in (0, 1024 // K - 1, 1024 // K, M - 1):
        A[i, rng.integers(K)] = [np.nan, np.inf][i % 2]
    B[K - 1, [0, N - 1]] = np.nan, -np.inf
    a, b = ia.Container.from_numpy(ctx, A, ch, bl), ia.Container.from_numpy(ctx, B, chb, (16, 8))
    c = ia.opt_gemm(ctx, a, b, (64, 16), (8, 8))
    got = c.to_numpy()
    ga, ach = O.encode_array(A, ch, bl)
    gb, bch = O.encode_array(B, chb, (16, 8))
    dt = O.DTYPE_DOUBLE if dtype is np.float64 else O.DTYPE_FLOAT
    ref = O.opt_gemm(ga, ach, gb, bch, O.Geom((M, N), (64, 16), (8, 8), A.itemsize), dt)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(got, ref)
    for x in (a, b, c):
        x.free()


def test_narrow_rows_cost_no_more_than_their_lines(ia):
    """8 million items as rows of 8 and as rows of 8000.  A narrow row's line of memory holds four
    times its items, and the scan's time is that of its lines: eight times leaves it room."""
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL)
    ms = {}
    for M, K in ((1_000_000, 8), (1000, 8000)):
        A = np.ones((M, K), np.float32)
        A[:500] = 0
        a = ia.Container.from_numpy(ctx, A, (M, K), (500, 8))
        b = ia.Container.from_numpy(ctx, np.ones((K, 8), np.float32), (K, 8), (8, 8))
        best = []
        for _ in range(4):
            ia.profile_kernels(True)
            ia.opt_gemm(ctx, a, b, (M, 8), (500, 8)).free()
            ctx.synchronize()
            ia.profile_kernels(False)
            best.append(ia.kernel_profile()["k_block_nonfinite"][1])
        ms[K] = min(best)
        a.free()
        b.free()
    assert ms[8] < 8 * ms[8000], ms
    ctx.close()
