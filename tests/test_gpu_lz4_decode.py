"""The LZ4 stream decoder on streams whose sequences meet its limits: windows (2048 compressed
bytes) that end at, just before and inside a sequence, the four tracks of a 32-byte segment
(3-byte sequences that keep their phase, literal runs that skip segments), match sources in the
window's output, in the 8 KiB ring, beyond it, self-overlapping ones, lengths around the
16- and 256-byte fill limits and the 3584-byte output group, and few long sequences.  Streams are
built token by token, so their contents do not depend on an encoder's choices."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _ext(v):
    out = bytearray()
    v -= 15
    while v >= 255:
        out.append(255)
        v -= 255
    out.append(v)
    return bytes(out)


def _stream(rng, size, lits, mls, dists):
    """(compressed, decoded): sequences with literal counts, match lengths and distances drawn
    from the lists until `size` decoded bytes, then the last literals."""
    comp, out = bytearray(), bytearray()
    while len(out) < size:
        lit, ml = max(int(rng.choice(lits)), 0 if out else 1), max(4, int(rng.choice(mls)))
        run = rng.integers(0, 256, lit).astype(np.uint8).tobytes()
        out += run
        d = min(int(rng.choice(dists)), len(out))
        comp.append((min(len(run), 15) << 4) | min(ml - 4, 15))
        if len(run) >= 15:
            comp += _ext(len(run))
        comp += run
        comp += bytes((d & 255, d >> 8))
        if ml - 4 >= 15:
            comp += _ext(ml - 4)
        src = len(out) - d
        if ml <= d:
            out += out[src:src + ml]
        else:
            out += (bytes(out[src:]) * (ml // d + 1))[:ml]
    last = rng.integers(0, 256, int(rng.integers(5, 40))).astype(np.uint8).tobytes()
    comp.append(min(len(last), 15) << 4)
    if len(last) >= 15:
        comp += _ext(len(last))
    comp += last
    out += last
    return bytes(comp), bytes(out)


CASES = {
    "three_byte": ([0], [4, 5, 6, 7], [1, 2, 3, 5, 40, 400, 3000]),
    "near": ([0, 1, 2], [4, 5, 9, 18], [1, 2, 3, 4, 5, 6, 7, 8, 9, 31]),
    "far": ([0, 1, 3], [4, 8, 15, 16, 17, 40], [4096, 8191, 8192, 8193, 12000, 40000, 65535]),
    "literals": ([0, 5, 14, 15, 16, 17, 31, 33, 60, 100], [4, 6, 19, 20], [1, 30, 500, 9000]),
    "lengths": ([0, 2, 13], [4, 12, 16, 17, 18, 19, 240, 255, 256, 257, 273, 274, 300], [7, 16, 200, 256, 300, 5000]),
    "long": ([0, 30, 269, 270, 271, 700, 2000, 2100, 5000], [4, 273, 274, 2000, 3583, 3584, 3585, 9000], [1, 3, 600, 8192, 20000]),
    "groups": ([0, 1], [500, 900, 1200, 3000], [1, 7, 400, 3500, 4700]),
}


@pytest.mark.parametrize("kind", sorted(CASES))
@pytest.mark.parametrize("size", [100, 3000, 70000])
def test_built_streams_decode(ctx, ia, kind, size):
    rng = np.random.default_rng(size)
    for seed in range(4):
        comp, want = _stream(rng, size, *CASES[kind])
        n = len(want)
        if len(comp) >= n:                                    # stored raw by the format's rules
            continue
        assert O.lz4_decompress(comp, n) == want
        # a chunk of one unsplit block of n bytes: header, bstart, csize, stream
        cbytes = 32 + 4 + 4 + len(comp)
        head = bytes([5, 1, 0x05 | 0x20 | 0x10, 1]) + n.to_bytes(4, "little") * 2 + cbytes.to_bytes(4, "little")
        head += bytes(6) + bytes([1]) + bytes(9)
        chunk = head + (36).to_bytes(4, "little") + len(comp).to_bytes(4, "little") + comp
        c = ia.Container.from_chunks(ctx, (n,), np.uint8, (n,), (n,), [chunk])
        got = c.to_numpy()
        want = np.frombuffer(want, np.uint8)
        assert np.array_equal(got, want), (kind, size, seed, int(np.argmax(got != want)))
        c.free()
