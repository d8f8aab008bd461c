"""The gather of blocks that share a CTA (fewer items than it has threads) and of blocks cut into several
slices, in single containers (the oracle's chunks) and in the batch, whose outputs are gathered by
one launch: rows of whole groups of 4 items and others, chunk and array padding."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

GEOMS = [
    ((37, 29), (10, 8), (1, 4)), ((37, 29), (10, 8), (3, 1)), ((37, 29), (10, 8), (5, 8)), ((61, 67), (32, 32), (8, 8)),
    ((100, 90), (32, 40), (4, 31)), ((100, 90), (32, 40), (4, 32)), ((100, 90), (33, 40), (16, 16)), ((300, 70), (64, 64), (32, 32)),
    ((40, 33), (20, 33), (3, 11)), ((200, 260), (200, 260), (129, 128)), ((200, 261), (200, 261), (128, 131)),
]


@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: "x".join(map(str, g[0] + g[2])))
@pytest.mark.parametrize("dtype", [np.float64, np.int32])
def test_blocks(ctx, ia, geom, dtype):
    shape, cs, bs = geom
    rng = np.random.default_rng(shape[0] * bs[1])
    x = (rng.standard_normal(shape) * 1000).astype(dtype)
    x[::3] = 5
    c = ia.Container.from_numpy(ctx, x, cs, bs)
    assert c.chunks() == O.encode_array(x, cs, bs)[1]
    c.free()


@pytest.mark.parametrize("block", [(8, 8), (5, 7), (128, 132), (129, 131), (200, 250)])
def test_batch_outputs(ia, block):
    """The batch's containers are those of the single products (whole numbers: every sum is exact)."""
    ctx = ia.Context()
    rng = np.random.default_rng(block[1])
    cs = (min(2 * block[0], 260), min(2 * block[1], 260))
    A, B, singles = [], [], []
    for m, k, n in ((261, 90, 270), (33, 41, 29), (200, 17, 250)):
        a = ia.Container.from_numpy(ctx, rng.integers(-64, 65, (m, k)).astype(np.float64), (cs[0], 50), (block[0], 25))
        b = ia.Container.from_numpy(ctx, rng.integers(-64, 65, (k, n)).astype(np.float64), (50, cs[1]), (25, block[1]))
        c = ia.opt_gemm(ctx, a, b, cs, block)
        singles.append(c.chunks())
        c.free()
        A.append(a)
        B.append(b)
    bt = ia.Batch(ctx, A, B, [cs] * 3, [block] * 3)
    for c, want in zip(bt.run(), singles):
        assert c.chunks() == want
        c.free()
    bt.free()
    ctx.close()
