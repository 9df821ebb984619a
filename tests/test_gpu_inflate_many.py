"""Many short streams decoded at once, by CTAs with smaller windows (4,608 bytes
of a stream), batches (1,024 tokens), pieces (2,048 bytes of output) and tables
(10 and 8 bits) than those a long stream gets: sizes and kinds around those cuts,
as members of one gzip file (decoded in parallel from 256 KiB on)."""
import random
import zlib

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu
STRATEGIES = [zlib.Z_DEFAULT_STRATEGY, zlib.Z_HUFFMAN_ONLY, zlib.Z_RLE, zlib.Z_FIXED]


def _member(d, level, strategy, flush_every=0):
    c = zlib.compressobj(level, zlib.DEFLATED, 31, 8, strategy)
    if not flush_every:
        return c.compress(d) + c.flush()
    return b"".join(c.compress(d[o:o + flush_every]) + c.flush(5) for o in range(0, len(d), flush_every)) + c.flush()


def _skewed(n, seed):
    """Symbols with Fibonacci counts (codes of up to 15 bits), matches at far distances."""
    counts = [1, 1]
    while sum(counts) < n:
        counts.append(counts[-1] + counts[-2])
    body = bytearray(b"".join(bytes([37 * i % 256]) * c for i, c in enumerate(counts)))[:n]
    random.Random(seed).shuffle(body)
    return bytes(body)


def _data(i, r):
    n = [1, 2, 33, 255, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4097, 5000, 8000][i % 14] + (i // 14) % 3
    if i % 9 == 0:
        return _skewed(min(n, 4000), i)
    if i % 50 == 7:
        return bytes(300000 + i)  # a short stream with much output
    if i % 11 == 3:
        unit = bytes(r.randrange(256) for _ in range(r.choice([1, 3, 31, 257, 259, 1500])))
        return (unit * (n // len(unit) + 2))[:n]
    return synth.gen(n, i % 6, i)


@pytest.mark.parametrize("count", [149, 400, 2700])
def test_members_around_the_cuts(gpu, count):
    r = random.Random(count)
    parts = [_data(i, r) for i in range(count)]
    packed = [_member(d, r.choice([1, 6, 9]), r.choice(STRATEGIES), r.choice([0, 0, 0, 90, 700])) for d in parts]
    if count < 2700:  # enough bytes for the parallel path: a last, long member
        parts.append(synth.gen(300000, 3, 1))
        packed.append(_member(parts[-1], 6, 0))
    data, file = b"".join(parts), b"".join(packed)
    assert len(file) >= 256 << 10
    assert gpu.decompress(file, gpu.Format.Gzip, len(data)) == data
    # a damaged member fails the file
    for k in (count // 3, count - 1):
        bad = [bytearray(p) for p in packed]
        bad[k][-12] ^= 0x10
        with pytest.raises(gpu.Error) as e:
            gpu.decompress(b"".join(map(bytes, bad)), gpu.Format.Gzip, len(data))
        assert e.value.code == -1
    with pytest.raises(gpu.Error):
        gpu.decompress(file, gpu.Format.Gzip, len(data) - 1)


@pytest.mark.parametrize("count, size", [(150, 60), (400, 150), (400, 3000), (3000, 1500)])
def test_batches_of_short_buffers_verify(gpu, count, size):
    import numpy as np
    parts = [synth.gen(1 + (size + 7 * i) % (2 * size), i % 6, i) for i in range(count)]
    data = np.frombuffer(b"".join(parts), np.uint8)
    for level in (0, 1, 6):
        b = gpu.DeviceBatch()
        b.load(data, [len(p) for p in parts], level, gpu.Format(1 + level % 2))
        b.run()
        b.sizes()
        assert all(b.verify())
        b.close()
