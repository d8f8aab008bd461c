"""The liblz4-identical encoder against the oracle's, byte for byte, where its 32-position
windows can go wrong: streams around the window, ring (2 KiB), fill (512 B) and table-kind
(65546 / 65547 B) edges, matches inside one window (short periods, runs), across windows and out
of the ring, literal runs and match lengths around the token's 15 and 255 steps."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = (12, 13, 14, 15, 31, 32, 33, 43, 44, 45, 63, 64, 65, 66, 97, 130, 511, 512, 545, 2047, 2048, 2083, 4099, 20000,
         65546, 65547, 70001)


def _streams(n):
    rng = np.random.default_rng(n)
    yield from (rng.integers(0, k, n) for k in (2, 3, 4, 6, 9, 16, 40, 256))
    yield from (np.minimum(rng.geometric(1 / k, n), 255) for k in (2, 5, 20))
    for period in (1, 2, 3, 5, 8, 29, 30, 31, 32, 33, 64, 300):
        x = np.tile(rng.integers(0, 256, period), n // period + 1)[:n]
        yield x
        y = x.copy()
        y[rng.integers(0, n, max(1, n // 40))] ^= 1
        yield y
    for gap in (3, 14, 15, 16, 18, 19, 20, 40, 269, 270, 271, 600, 3000):   # literals or matches of that length
        x = rng.integers(0, 256, n)
        unit = rng.integers(0, 256, gap + 8)
        for a in range(gap, n - len(unit), 2 * gap + 9):
            x[a:a + gap] = unit[:gap]
        yield x
    x = np.zeros(n, int)
    x[rng.integers(0, n, max(1, n // 200))] = 9
    yield x


@pytest.mark.parametrize("n", SIZES)
def test_streams_equal_the_oracles(ctx, ia, n):
    for i, x in enumerate(_streams(n)):
        x = x.astype(np.uint8)
        c = ia.Container.from_numpy(ctx, x, (n,), (n,))
        _, want = O.encode_array(x, (n,), (n,))
        assert c.chunks() == want, (n, i)
        c.free()


@pytest.mark.parametrize("n", range(1, 15))
def test_parallel_encoder_streams_below_its_probe(ia, n):
    """Streams of a few bytes: shorter than the 13 bytes LZ4 compresses and the 11 the probe of
    the parallel encoder reads at a time; they are stored raw."""
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL)
    x = np.random.default_rng(n).integers(0, 256, 7 * n).astype(np.uint8)
    c = ia.Container.from_numpy(ctx, x, (7 * n,), (n,))
    _, want = O.encode_array(x, (7 * n,), (n,))
    assert c.chunks() == want
    assert np.array_equal(c.to_numpy(), x)
    c.free()
    ctx.close()
