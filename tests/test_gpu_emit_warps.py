"""Chunks whose streams are written by a warp each (more streams than CTAs run at once, each below 8 KiB)
and by a CTA each, around both limits, against the oracle's: raw, LZ4 and run streams, chunks stored as
they are, compression level 0.  The batch writes its outputs' streams by the same rule."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def values(n, dtype, seed):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal(n) * 1000).astype(dtype)
    x[:n // 3] = np.arange(n // 3) // 7
    x[n // 3:n // 2] = 3
    return x


@pytest.mark.parametrize("dtype,block,count", [
    (np.float64, 33, 160), (np.float64, 64, 147), (np.float64, 64, 149), (np.float32, 1024, 300),
    (np.uint8, 8191, 1183), (np.uint8, 8191, 1185), (np.uint8, 8192, 1185), (np.float64, 8191, 150), (np.float64, 8192, 150),
])
@pytest.mark.parametrize("level", [5, 0])
def test_streams(ia, dtype, block, count, level):
    cfg = ia.Config.defaults()
    cfg.compression_level = level
    ctx = ia.Context(cfg)
    x = values(block * count - 5, dtype, block)
    chunk = block * 40
    c = ia.Container.from_numpy(ctx, x, (chunk,), (block,))
    got = c.chunks()
    if level:
        assert got == O.encode_array(x, (chunk,), (block,))[1]
    else:
        assert all(k[2] & 2 and len(k) == 32 + chunk * x.itemsize for k in got)
    assert np.array_equal(c.to_numpy(), x)
    c.free()
    ctx.close()


@pytest.mark.parametrize("block", [(6, 8), (90, 91)])
def test_batch(ia, block):
    ctx = ia.Context()
    rng = np.random.default_rng(5)
    cs = (4 * block[0], 3 * block[1])
    A, B, singles = [], [], []
    for m, k, n in ((300, 20, 310), (170, 31, 400)):
        a = ia.Container.from_numpy(ctx, rng.integers(-64, 65, (m, k)).astype(np.float64), (cs[0], 16), (block[0], 8))
        b = ia.Container.from_numpy(ctx, rng.integers(-64, 65, (k, n)).astype(np.float64), (16, cs[1]), (8, block[1]))
        c = ia.opt_gemm(ctx, a, b, cs, block)
        singles.append(c.chunks())
        assert singles[-1] == O.encode_array(c.to_numpy(), cs, block)[1]
        c.free()
        A.append(a)
        B.append(b)
    bt = ia.Batch(ctx, A, B, [cs] * 2, [block] * 2)
    for c, want in zip(bt.run(), singles):
        assert c.chunks() == want
        c.free()
    bt.free()
    ctx.close()


def test_short_streams_cost_no_cta_each(ia):
    """2 million streams of 64 bytes against 1,024 times as long ones of the same bytes: the launch is
    bound by the streams' loads, which a warp each keeps under way (0.8 ms; a CTA each 3.6)."""
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL)
    x = np.random.default_rng(1).standard_normal((4000, 4000))
    ms = {}
    for b in (8, 250):
        times = []
        for _ in range(3):
            ia.profile_kernels(True)
            ia.Container.from_numpy(ctx, x, (1000, 1000), (b, b)).free()
            ctx.synchronize()
            ia.profile_kernels(False)
            times.append(ia.kernel_profile()["k_emit"][1])
        ms[b] = min(times)
    assert ms[8] < 40 * ms[250], ms
    ctx.close()
