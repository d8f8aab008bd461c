"""The larger tiles of the native products (float64 64 x 64, float32 128 x 128) at ragged rows, columns
and k steps, also where zero-block pairs are left out.  The sizes are just below one tile for each
multiprocessor, which is where the larger tile is taken; the rule is restated here so that a
change of it does not leave these tiles untested.  Whole numbers make every sum exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def takes_larger(tile, m, n, sms):
    def busiest(t):
        return -(-(-(-m // t) * -(-n // t)) // sms) * t * t
    small, extra = tile // 2, 11 if tile == 64 else 14
    return not busiest(small) * extra < busiest(tile) * 10


def sizes(tile, sms):
    side = int(sms ** 0.5)
    for m, n in ((side * tile - 1, side * tile - tile + 1), (side * tile - tile + 33, side * tile), (side * tile, side * tile - 2)):
        assert takes_larger(tile, m, n, sms)
        yield m, n


@pytest.mark.parametrize("dtype,tile", [(np.float64, 64), (np.float32, 128)])
@pytest.mark.parametrize("k", [1, 7, 8, 31, 33, 70, 129])
def test_ragged(ia, ctx, dtype, tile, k):
    import torch
    td = torch.float64 if dtype is np.float64 else torch.float32
    rng = np.random.default_rng(k)
    for m, n in sizes(tile, torch.cuda.get_device_properties(0).multi_processor_count):
        a, b = rng.integers(-64, 65, (m, k)).astype(dtype), rng.integers(-64, 65, (k, n)).astype(dtype)
        up = lambda v: -(-v // 4) * 4  # noqa: E731
        A = torch.full((m, up(k)), float("nan"), dtype=td, device="cuda")     # padding is never read
        B = torch.full((k, up(n)), float("nan"), dtype=td, device="cuda")
        C = torch.full((m, up(n) + 4), 3.0, dtype=td, device="cuda")
        A[:, :k] = torch.from_numpy(a).cuda()
        B[:, :n] = torch.from_numpy(b).cuda()
        torch.cuda.synchronize()
        ia.check(ia.lib().iarray_b200_dense_gemm(ctx.ptr, 0 if dtype is np.float64 else 1, m, n, k, A.data_ptr(),
                                                 A.stride(0), B.data_ptr(), B.stride(0), C.data_ptr(), C.stride(0)))
        ctx.synchronize()
        got = C.cpu().numpy()
        assert np.array_equal(got[:, :n], a @ b), (m, n)
        assert np.all(got[:, n:] == 3.0), (m, n)


@pytest.mark.parametrize("dtype,tile", [(np.float64, 64), (np.float32, 128)])
def test_zero_block_pairs(ia, ctx, dtype, tile):
    import torch
    rng = np.random.default_rng(tile)
    for m, n in sizes(tile, torch.cuda.get_device_properties(0).multi_processor_count):
        k, block = 333, 32
        A, B = rng.integers(-64, 65, (m, k)).astype(dtype), rng.integers(-64, 65, (k, n)).astype(dtype)
        for x in (A, B):                                    # six of ten blocks are zero, and whole k ranges
            keep = rng.random((-(-x.shape[0] // block), -(-x.shape[1] // block))) < 0.4
            x *= np.kron(keep, np.ones((block, block)))[:x.shape[0], :x.shape[1]].astype(dtype)
        A[:, 64:128] = 0
        B[192:224] = 0
        a = ia.Container.from_numpy(ctx, A, (256, 256), (block, block))
        b = ia.Container.from_numpy(ctx, B, (256, 256), (block, block))
        c = ia.opt_gemm(ctx, a, b, (256, 256), (block, block))
        assert np.array_equal(c.to_numpy(), A @ B), (m, n)
        for x in (a, b, c):
            x.free()
