"""The parallel-parse encoder against its rule restated position by position, byte for byte: match
lengths around 16 bytes and the cap of 128, runs whose candidate lies in a shorter, longer or equally
long run, rows of positions with one distance and many rows side by side, literal runs around 16 and
the token's 15 and 255 steps, windows (1024) and rounds (32, 128, 256), candidates inside and
outside the 4 KiB window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 128


def model(x):
    """One stream: the greedy parse over every position's longest of two candidates, the latest
    position of its hash bucket before its round and, in a run, the previous position."""
    x = bytes(x)
    n = len(x)

    def common(p, c, most):
        k = 0
        while k < most and x[p + k] == x[c + k]:
            k += 1
        return k

    table, length, dist = {}, [0] * n, [0] * n
    p, first = 0, n - 11
    while p < first:
        size = 32 if p < 128 else 128 if p < 256 else 256
        entered = {}
        for q in range(p, min(p + size, first)):
            h = (int.from_bytes(x[q:q + 4], "little") * 2654435761 % 2**32) >> 20
            c, most = table.get(h, -1), min(n - 5 - q, CAP)
            if c >= 0 and q - c <= 65535 and x[c:c + 4] == x[q:q + 4]:
                length[q], dist[q] = common(q, c, most), q - c
            if q and c != q - 1 and x[q - 1:q + 3] == x[q:q + 4]:
                k = common(q, q - 1, most)
                if k > length[q]:
                    length[q], dist[q] = k, 1
            entered[h] = q
        table.update(entered)
        p += size
    out, anchor, p = bytearray(), 0, 0

    def extra(v):
        return bytes([255] * ((v - 15) // 255) + [(v - 15) % 255]) if v >= 15 else b""

    while p < first:
        if length[p] < 4:
            p += 1
            continue
        k = length[p] if length[p] < CAP else common(p, p - dist[p], n - 5 - p)
        lit = p - anchor
        out += bytes([min(lit, 15) << 4 | min(k - 4, 15)]) + extra(lit) + x[anchor:p] + dist[p].to_bytes(2, "little")
        out += extra(k - 4)
        p = anchor = p + k
    lit = n - anchor
    return bytes(out + bytes([min(lit, 15) << 4]) + extra(lit) + x[anchor:])


def streams(n):
    rng = np.random.default_rng(n)
    for k in (2, 3, 5):
        yield rng.integers(0, k, n)
    for lo, hi in ((3, 40), (10, 20), (100, 160), (200, 900)):         # runs, one after the other
        w = rng.integers(lo, hi, n // lo + 2)
        yield np.repeat(rng.integers(0, 3, len(w)), w)[:n]
    for run in (15, 16, 17, 33, 127, 128, 129, 300):                    # equal runs apart
        x = np.tile(np.concatenate([np.zeros(run, int), [1, 2, 3, 1, 7]]), n // run + 1)[:n]
        yield x
        y = x.copy()
        y[rng.integers(0, n, n // 100)] ^= 1
        yield y
    for unit, gap in ((5, 14), (18, 3), (40, 15), (40, 16), (40, 17), (140, 33), (300, 270)):   # repeats between noise
        words = [rng.integers(0, 256, unit) for _ in range(7)]
        parts = []
        while sum(map(len, parts)) < n:
            parts += [words[rng.integers(7)], words[rng.integers(7)], rng.integers(0, 256, gap)]
        yield np.concatenate(parts)[:n]
    x = np.zeros(n, int)
    x[::128] = rng.integers(0, 256, len(x[::128]))                      # rows of noise and zeros
    x.reshape(-1)[:n // 128 * 128].reshape(-1, 128)[:, :50] = rng.integers(0, 256, (n // 128, 50))
    yield x


@pytest.mark.parametrize("n", [1024, 1035, 2047, 2060, 4500, 20011])
def test_streams_equal_the_rules(ia, n):
    ctx, exact = ia.Context(encoder=ia.ENCODER_PARALLEL), ia.Context()
    parsed = 0
    for i, x in enumerate(streams(n)):
        x = x.astype(np.uint8)
        c = ia.Container.from_numpy(ctx, x, (n,), (n,))
        assert np.array_equal(c.to_numpy(), x), (n, i)
        chunk, = c.chunks()
        c.free()
        at = int.from_bytes(chunk[32:36], "little")
        size = int.from_bytes(chunk[at:at + 4], "little", signed=True)
        if chunk[2] & 2 or size <= 0 or size == n:
            continue                                                    # a run, or stored raw
        if chunk[at + 4:at + 4 + size] == model(x):
            parsed += 1
            continue
        c = ia.Container.from_numpy(exact, x, (n,), (n,))               # few matches: the liblz4 search
        assert c.chunks() == [chunk], (n, i)
        c.free()
    assert parsed >= 20
    exact.close()
    ctx.close()
