"""iarray_b200_opt_gemm_cframes with the default (liblz4-identical) encoder, whose bands are
encoded side by side: one band, as many as there are encode streams, more, and ragged last
bands; the frame equals the sequential calls' byte for byte, twice in a row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bands,last", [(1, 40), (4, 40), (5, 40), (9, 7)])
@pytest.mark.parametrize("form", ["native", "split"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_bands(ia, bands, last, form, dtype):
    ctx = ia.Context(form=ia.FORM_SPLIT if form == "split" else ia.FORM_NATIVE)
    rng = np.random.default_rng(bands)
    M, K, N = (bands - 1) * 40 + last, 90, 130
    A = (rng.uniform(-1, 1, (M, K)) * np.exp2(rng.integers(-8, 9, (M, K)))).astype(dtype)
    B = rng.uniform(-1, 1, (K, N)).astype(dtype)
    fa = ia.Container.from_numpy(ctx, A, (40, 50), (20, 25)).to_cframe()
    fb = ia.Container.from_numpy(ctx, B, (50, 64), (25, 32)).to_cframe()
    c = ia.opt_gemm(ctx, ia.Container.from_cframe(ctx, fa), ia.Container.from_cframe(ctx, fb), (40, 64), (20, 32))
    want = c.to_cframe()
    for _ in range(2):
        out, n = ia.opt_gemm_cframes(ctx, fa, fb, (40, 64), (20, 32))
        assert out[:n].tobytes() == want
    ctx.close()
