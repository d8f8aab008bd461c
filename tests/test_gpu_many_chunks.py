"""The chunk offsets of encoded containers around the counts where they get a launch of their own (more
than 1024 chunks) and where that launch takes another round (8192 chunks): the chunks are the
oracle's, and the decoder finds them by the device's index."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 1024, 1025, 8191, 8192, 8193, 20011])
@pytest.mark.parametrize("encoder", ["liblz4", "parallel"])
def test_chunks(ia, n, encoder):
    ctx = ia.Context(encoder=ia.ENCODER_PARALLEL if encoder == "parallel" else ia.ENCODER_LIBLZ4)
    x = (np.random.default_rng(n).standard_normal(40 * n - 7) * 100).astype(np.float32)
    x[::3] = 1
    x[: 40 * (n // 5)] = 2                                      # chunks of several sizes
    c = ia.Container.from_numpy(ctx, x, (40,), (20,))
    assert np.array_equal(c.to_numpy(), x)
    if encoder == "liblz4":
        assert c.chunks() == O.encode_array(x, (40,), (20,))[1]
    back = ia.Container.from_cframe(ctx, c.to_cframe())
    assert np.array_equal(back.to_numpy(), x)
    back.free()
    c.free()
    ctx.close()
