"""Streams of many short blocks: the decoder keeps staged words, the fixed
code's tables and the last block's size from one block to the next."""
import random
import zlib

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu

BLOCK = 5  # Z_BLOCK: ends a block without aligning to a byte


def _stream(sizes, kinds, strategies, flushes, seed):
    """One raw stream of segments (each one deflater's, so their codes differ) of blocks of the given sizes."""
    rng = random.Random(seed)
    data, out = b"", b""
    for seg in range(4):
        c = zlib.compressobj(rng.choice([1, 6, 9]), zlib.DEFLATED, -15, 8, rng.choice(strategies))
        for i in range(60):
            d = synth.gen(rng.choice(sizes), rng.choice(kinds), 1000 * seed + 100 * seg + i)
            data += d
            out += c.compress(d) + c.flush(rng.choice(flushes))
        out += c.flush(zlib.Z_FULL_FLUSH if seg < 3 else zlib.Z_FINISH)
    assert zlib.decompress(out, -15) == data
    return data, out


FIXED, DYNAMIC = [zlib.Z_FIXED], [zlib.Z_DEFAULT_STRATEGY, zlib.Z_HUFFMAN_ONLY]


@pytest.mark.parametrize("sizes", [[1, 3, 100], [0, 40, 1000], [5, 9000], [100, 60000, 120000], [36800, 36900, 1]])
@pytest.mark.parametrize("strategies", [FIXED, DYNAMIC, FIXED + DYNAMIC])
def test_short_and_long_blocks(gpu, sizes, strategies):
    for seed in range(3):
        flushes = [[BLOCK], [zlib.Z_SYNC_FLUSH, BLOCK], [zlib.Z_PARTIAL_FLUSH, zlib.Z_FULL_FLUSH]][seed]
        data, out = _stream(sizes, [0, 1, 3, 5], strategies, flushes, 17 * seed + len(sizes))
        assert gpu.decompress(out, gpu.Format.Raw, len(data)) == data
        with pytest.raises(gpu.Error):
            gpu.decompress(out[:-1], gpu.Format.Raw, len(data))
        if data:
            with pytest.raises(gpu.Error):
                gpu.decompress(out, gpu.Format.Raw, len(data) - 1)


def test_tables_of_one_stream_do_not_serve_the_next(gpu):
    """Streams of one launch, fixed and dynamic in turn, that the same CTAs decode."""
    import gzip
    import numpy as np
    parts, packed = [], []
    for i in range(1200):
        d = synth.gen(300 + 13 * i % 1500, i % 4, i)
        c = zlib.compressobj(6, zlib.DEFLATED, 31, 8, zlib.Z_FIXED if i % 3 else zlib.Z_DEFAULT_STRATEGY)
        parts.append(d)
        packed.append(c.compress(d) + c.flush())
    data = b"".join(parts)
    assert gzip.decompress(b"".join(packed)) == data
    assert gpu.decompress(b"".join(packed), gpu.Format.Gzip, len(data)) == data
    b = gpu.DeviceBatch()
    for level in (1, 6):  # fixed, then dynamic and stored
        b.load(np.frombuffer(data, np.uint8), [len(p) for p in parts], level, gpu.Format.Zlib)
        b.run()
        b.sizes()
        assert all(b.verify())
    b.close()
