"""Products of more rows than 65535 row tiles.  Whole-number operands make every sum exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows past 65535 tiles of 32 (float64, at most 32 columns) and of 64 rows (float32)
TALL = [(np.float64, 2_100_000), (np.float32, 4_200_000)]


def operands(dtype, M):
    rng = np.random.default_rng(M)
    return rng.integers(-8, 9, (M, 8)).astype(dtype), rng.integers(-8, 9, (8, 8)).astype(dtype)


@pytest.mark.parametrize("dtype,M", TALL)
def test_one_band_of_frames(ia, dtype, M):
    """A band whose product cannot be launched must not come back as a frame."""
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL)
    A, B = operands(dtype, M)
    fa = ia.Container.from_numpy(ctx, A, (M, 8), (M // 1000, 8)).to_cframe()
    fb = ia.Container.from_numpy(ctx, B, (8, 8), (8, 8)).to_cframe()
    try:
        out, n = ia.opt_gemm_cframes(ctx, fa, fb, (M, 8), (M // 1000, 8))
    except ia.IArrayError as e:
        assert e.name == "GPU_FAILED"
    else:
        c = ia.Container.from_cframe(ctx, out[:n].tobytes())
        assert np.array_equal(c.to_numpy(), A @ B)
    ctx.close()
