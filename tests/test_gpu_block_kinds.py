"""Decoding containers whose blocks are of different kinds side by side (split planes, raw planes,
runs, stored raw, zero chunks), below and above the size from which the blocks that are not split
by bytes get a launch of their own, with ragged edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOMS = [
    ((301, 259), (100, 130), (50, 65)),
    ((40, 24), (20, 12), (20, 12)),                # one block a chunk, one warp of blocks
    ((4099, 4111), (1024, 1028), (256, 257)),      # 64 MiB and more of 4-byte items
]
DTYPES = [np.float64, np.float32, np.int32, np.uint8]


def kinds(shape, cs, dtype):
    """Chunks in turn smooth, random, zero, constant, and with random low bytes."""
    rng = np.random.default_rng(7)
    x = (np.arange(shape[0], dtype=np.float64)[:, None] * 3 + np.arange(shape[1])).astype(dtype)
    k = 0
    for i in range(0, shape[0], cs[0]):
        for j in range(0, shape[1], cs[1]):
            t = x[i:i + cs[0], j:j + cs[1]]
            if k % 5 == 1:
                t[...] = rng.integers(0, 120, t.shape + (t.itemsize,), dtype=np.uint8).view(dtype)[..., 0]
            elif k % 5 == 2:
                t[...] = 0
            elif k % 5 == 3:
                t[...] = 77
            elif k % 5 == 4:
                t[...] = t + rng.integers(0, 100, t.shape).astype(dtype)
            k += 1
    return x


@pytest.mark.parametrize("geom", GEOMS, ids=lambda g: "x".join(map(str, g[0])))
@pytest.mark.parametrize("dtype", DTYPES)
def test_kinds_side_by_side(ctx, ia, geom, dtype):
    shape, cs, bs = geom
    x = kinds(shape, cs, dtype)
    c = ia.Container.from_numpy(ctx, x, cs, bs)
    assert np.array_equal(c.to_numpy().view(np.uint8), x.view(np.uint8))
    c.free()
