"""Containers of which no block, some or every block takes the general scatter, which the parse counts:
blocks stored as they are, unsplit, special and zero chunks beside split ones, of 1- to 8-byte items,
through the allocating decoder, the pair decode of the products and the one without allocation."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def container(ia, level, split, dtype, shape, cs, bs):
    cfg = ia.Config.defaults()
    cfg.compression_level = level
    if split is not None:
        cfg.splitmode = split
    ctx = ia.Context(cfg)
    rng = np.random.default_rng(shape[0])
    x = (rng.standard_normal(shape) * 50).astype(dtype)
    x[: shape[0] // 2, : shape[1] // 2] = 3                           # compressible chunks beside raw ones
    return ctx, x, ia.Container.from_numpy(ctx, x, cs, bs)


@pytest.mark.parametrize("level,split", [(0, None), (5, None), (5, 1), (5, 2)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int16, np.uint8])
@pytest.mark.parametrize("geom", [((200, 200), (200, 200), (100, 200)), ((301, 259), (100, 130), (50, 65)), ((64, 60), (16, 20), (4, 5)),
                                  ((97, 3001), (97, 1024), (97, 513))], ids=lambda g: "x".join(map(str, g[0])))
def test_decode(ia, level, split, dtype, geom):
    import torch
    shape, cs, bs = geom
    ctx, x, c = container(ia, level, split, dtype, shape, cs, bs)
    assert np.array_equal(c.to_numpy(), x)
    chunks = b"".join(c.chunks())
    dev = torch.from_numpy(np.frombuffer(chunks, np.uint8).copy()).cuda()
    out = torch.zeros(x.nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    I64 = ctypes.c_int64 * 2
    rc = ia.lib().iarray_b200_decode_noalloc(2, I64(*shape), I64(*cs), I64(*bs), x.itemsize, dev.data_ptr(), len(chunks),
                                             out.data_ptr(), shape[1], None)
    ia.check(rc)
    assert np.array_equal(out.cpu().numpy().view(dtype).reshape(shape), x)
    c.free()
    ctx.close()


@pytest.mark.parametrize("level", [0, 5])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_product(ia, level, dtype):
    cfg = ia.Config.defaults()
    cfg.compression_level = level
    ctx, plain = ia.Context(cfg), ia.Context()
    rng = np.random.default_rng(3)
    A, B = rng.integers(-64, 65, (130, 77)).astype(dtype), rng.integers(-64, 65, (77, 99)).astype(dtype)
    A[:32, :32] = 0
    a, b = ia.Container.from_numpy(ctx, A, (64, 64), (32, 32)), ia.Container.from_numpy(plain, B, (64, 64), (32, 32))
    c = ia.opt_gemm(ctx, a, b, (64, 64), (32, 32))
    assert np.array_equal(c.to_numpy(), A @ B)
    for x in (a, b, c):
        x.free()
    ctx.close()
    plain.close()
