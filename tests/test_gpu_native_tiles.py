"""The native dense products at the edges of their tiles (float64 32 x 32 and 64 x 64, float32
64 x 64 and 128 x 128) and k steps.  Operands are small whole numbers, so every sum is exact and
the result must equal the whole-number product; columns past N keep their contents."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200]
SIZES = [(m, EDGES[(i * 7 + 3) % len(EDGES)], k) for i, m in enumerate(EDGES) for k in (1, 7, 8, 9, 17, 33, 70)]
# enough tiles for the larger shape of each type
SIZES += [(1100, 1165, 40), (1601, 1500, 9)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_tiles(ia, ctx, dtype):
    import torch
    td = torch.float64 if dtype is np.float64 else torch.float32
    rng = np.random.default_rng(5)
    for m, n, k in SIZES:
        a = rng.integers(-64, 65, (m, k))
        b = rng.integers(-64, 65, (k, n))
        up = lambda v: -(-v // 4) * 4  # noqa: E731
        A = torch.full((m, up(k)), float("nan"), dtype=td, device="cuda")     # padding is never read
        B = torch.full((k, up(n)), float("nan"), dtype=td, device="cuda")
        C = torch.full((m, up(n) + 4), 3.0, dtype=td, device="cuda")
        A[:, :k] = torch.from_numpy(a.astype(dtype)).cuda()
        B[:, :n] = torch.from_numpy(b.astype(dtype)).cuda()
        torch.cuda.synchronize()
        ia.check(ia.lib().iarray_b200_dense_gemm(ctx.ptr, 0 if dtype is np.float64 else 1, m, n, k, A.data_ptr(),
                                                 A.stride(0), B.data_ptr(), B.stride(0), C.data_ptr(), C.stride(0)))
        ctx.synchronize()
        got = C.cpu().numpy()
        assert np.array_equal(got[:, :n], (a @ b).astype(dtype)), (m, n, k)
        assert np.all(got[:, n:] == 3.0), (m, n, k)
