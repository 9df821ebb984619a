"""Decoding at the edges of what the inflate kernel cuts a stream into: parts of
288 bits and windows of 36 KiB of the stream, batches of 8,192 tokens, pieces
of 16 KiB of output; matches that repeat themselves across them; many small
blocks; and damaged streams, which must fail or decode exactly as zlib does."""
import random
import zlib

import pytest

from orot_b200 import deflate, synth

pytestmark = pytest.mark.gpu
STRATEGIES = [zlib.Z_DEFAULT_STRATEGY, zlib.Z_HUFFMAN_ONLY, zlib.Z_RLE, zlib.Z_FIXED]


def pack(data, level=6, strategy=0, mem=8, flush_every=0, mode=zlib.Z_FULL_FLUSH):
    c = zlib.compressobj(level, zlib.DEFLATED, -15, mem, strategy)
    if not flush_every:
        return c.compress(data) + c.flush()
    out = b"".join(c.compress(data[o:o + flush_every]) + c.flush(mode) for o in range(0, len(data), flush_every))
    return out + c.flush()


def check(stream, data):
    assert deflate.decompress(stream, deflate.Format.Raw, len(data)) == data


@pytest.mark.parametrize("n", [1, 2, 287, 289, 8191, 8192, 8193, 16383, 16384, 16385, 32769, 36864, 65537, 300001])
def test_sizes_around_the_cuts(gpu, n):
    for kind in range(6):
        d = synth.gen(n, kind, n + kind)
        for strategy in STRATEGIES:
            check(pack(d, strategy=strategy), d)


@pytest.mark.parametrize("period", [1, 2, 3, 7, 31, 257, 258, 259, 16383, 16384, 32768])
def test_matches_that_repeat_themselves(gpu, period):
    r = random.Random(period)
    unit = bytes(r.randrange(256) for _ in range(period))
    for n in (period + 300, 20000 + period, 16384 * 3 + 5):
        d = (unit * (n // period + 1))[:n]
        check(pack(d, 9), d)
        d = bytes(r.randrange(256) for _ in range(100)) + d + b"end"
        check(pack(d, 9), d)


def test_long_codes_and_skewed_symbols(gpu):
    """Fibonacci counts give codes of up to 15 bits; each symbol also alone."""
    counts = [1, 1]
    while len(counts) < 22:
        counts.append(counts[-1] + counts[-2])
    body = bytearray(b"".join(bytes([i]) * c for i, c in enumerate(counts)))
    random.Random(1).shuffle(body)
    d = bytes(body)
    check(pack(d, strategy=zlib.Z_HUFFMAN_ONLY), d)
    check(pack(d), d)


@pytest.mark.parametrize("every", [1, 100, 4096, 70000])
def test_many_blocks(gpu, every):
    d = synth.gen(40 * every if every < 4096 else 300000, synth.MIXED if every > 4096 else synth.TEXT, every)
    for mode in (zlib.Z_FULL_FLUSH, zlib.Z_SYNC_FLUSH):
        check(pack(d, 6, 0, 8, every, mode), d)
    check(pack(d, 6, 0, 1), d)  # the smallest blocks zlib makes


@pytest.mark.parametrize("seed", range(6))
def test_damaged_streams_fail_as_in_zlib(gpu, seed):
    r = random.Random(seed)
    d = synth.gen(60000, seed, seed)
    good = pack(d, r.choice([1, 6, 9]), r.choice(STRATEGIES))
    for _ in range(40):
        bad = bytearray(good[:r.randrange(1, len(good))] if r.random() < 0.3 else good)
        for _ in range(r.randrange(1, 4)):
            bad[r.randrange(len(bad))] ^= 1 << r.randrange(8)
        z = zlib.decompressobj(-15)
        try:
            want = z.decompress(bytes(bad)) + z.flush()
            if not z.eof:
                want = None
        except zlib.error:
            want = None
        try:
            got = deflate.decompress(bytes(bad), deflate.Format.Raw, 4 << 20)
        except deflate.Error as e:
            assert e.code == -1
            got = None
        # zlib also rejects codes that are not complete; a stream that meets
        # none of the unassigned ones decodes here, as in the reference
        assert got == want or (want is None and got is not None)
