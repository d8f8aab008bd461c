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


@pytest.mark.parametrize("dtype,M", TALL)
@pytest.mark.parametrize("zeros", [False, True])
def test_containers_and_frames(ia, dtype, M, zeros):
    """(With a zero block the float64 product is the kernel that leaves out zero-block pairs.)"""
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL)
    A, B = operands(dtype, M)
    block = (M // 1000, 8)
    if zeros:
        A[-2 * block[0]:-block[0]] = 0
    want = A @ B
    a, b = ia.Container.from_numpy(ctx, A, (M, 8), block), ia.Container.from_numpy(ctx, B, (8, 8), (8, 8))
    for product in (ia.opt_gemm, ia.matmul):
        c = product(ctx, a, b, (M, 8), block)
        assert np.array_equal(c.to_numpy(), want)
        c.free()
    out, n = ia.opt_gemm_cframes(ctx, a.to_cframe(), b.to_cframe(), (M, 8), block)
    c = ia.Container.from_cframe(ctx, out[:n].tobytes())
    assert np.array_equal(c.to_numpy(), want)
    ctx.close()


@pytest.mark.parametrize("dtype,M,N", [
    (np.float64, 65535 * 32, 16), (np.float64, 65535 * 32 + 1, 16), (np.float64, 2 * 65535 * 32 + 33, 8),
    (np.float64, 65535 * 64 + 1, 40),                        # 64-row tiles
    (np.float32, 65535 * 64, 16), (np.float32, 65535 * 64 + 1, 16), (np.float32, 8_388_480, 4),
])
def test_dense_rows(ia, ctx, dtype, M, N):
    import torch
    td = torch.float64 if dtype is np.float64 else torch.float32
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    A = torch.randint(-8, 9, (M, 4), generator=g, device="cuda").to(td)
    B = torch.randint(-8, 9, (4, N), generator=g, device="cuda").to(td)
    C = torch.full((M, N), 7.0, dtype=td, device="cuda")
    torch.cuda.synchronize()
    ia.check(ia.lib().iarray_b200_dense_gemm(ctx.ptr, 0 if dtype is np.float64 else 1, M, N, 4, A.data_ptr(), 4,
                                             B.data_ptr(), N, C.data_ptr(), N))
    ctx.synchronize()
    assert torch.equal(C, sum(A[:, k:k + 1] * B[k:k + 1] for k in range(4)))
