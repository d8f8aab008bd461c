"""Streams of one byte value and those that differ from one in a single byte, for both encoders: the
check reads 16-byte words, the bytes before the first whole word and after the last by themselves.
Blocks of odd sizes put the streams at every alignment."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [13, 15, 16, 17, 31, 33, 47, 1023, 2047, 2048, 2049, 8191, 8193, 20011])
def test_one_byte_apart(ia, ctx, n):
    """One stream (a block of n bytes) after the other, each with its odd byte elsewhere, or none."""
    at = sorted({0, 1, 14, 15, 16, 17, n // 2, n - 18, n - 17, n - 16, n - 2, n - 1} & set(range(n)))
    x = np.full((len(at) + 1, n), 7, np.uint8)
    for row, p in zip(x, at):
        row[p] = 8
    x = x.reshape(-1)
    _, want = O.encode_array(x, x.shape, (n,))
    c = ia.Container.from_numpy(ctx, x, x.shape, (n,))
    assert c.chunks() == want
    c.free()
    par = ia.Context(encoder=ia.ENCODER_PARALLEL)
    c = ia.Container.from_numpy(par, x, x.shape, (n,))
    assert np.array_equal(c.to_numpy(), x)
    chunk, = c.chunks()
    if not chunk[2] & 2:                                            # (not stored as it is)
        for b in range(len(at) + 1):
            p = int.from_bytes(chunk[32 + 4 * b:36 + 4 * b], "little")
            size = int.from_bytes(chunk[p:p + 4], "little", signed=True)
            assert (size < 0) == (b == len(at)), b                  # a run only where no byte differs
    c.free()
    par.close()
