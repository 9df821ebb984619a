"""Damaged streams: the GPU decoder must give what a plain decoder written from RFC
1951 gives, bytes or an error.  (zlib also rejects every code that is not complete;
the engine, like the reference, only one that is met unassigned.)  And outputs
larger than the pinned staging they are fetched through."""
import gzip
import random
import zlib

import numpy as np
import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu

ORDER = [16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15]


class Bad(Exception):
    pass


def _code(lengths):
    """{(length, code): symbol}, codes most significant bit first; over-subscribed sets are refused."""
    left = 1
    for n in range(1, 16):
        left = 2 * left - lengths.count(n)
        if left < 0:
            raise Bad("over-subscribed")
    table, code = {}, 0
    for n in range(1, 16):
        for s, k in enumerate(lengths):
            if k == n:
                table[n, code] = s
                code += 1
        code <<= 1
    return table


def plain_inflate(z, cap):
    """RFC 1951, one bit at a time."""
    bits = "".join(f"{b:08b}"[::-1] for b in z)
    pos, out = 0, bytearray()

    def take(n):
        nonlocal pos
        if pos + n > len(bits):
            raise Bad("input ends")
        v = int(bits[pos:pos + n][::-1], 2) if n else 0
        pos += n
        return v

    def symbol(table):
        code = 0
        for n in range(1, 16):
            code = 2 * code + take(1)
            if (n, code) in table:
                return table[n, code]
        raise Bad("unassigned code")

    last = 0
    while not last:
        last, kind = take(1), take(2)
        if kind == 3:
            raise Bad("block type")
        if kind == 0:
            pos = (pos + 7) // 8 * 8
            n, inv = take(16), take(16)
            if n ^ inv != 0xFFFF or pos + 8 * n > len(bits):
                raise Bad("stored block")
            out += z[pos // 8:pos // 8 + n]
            pos += 8 * n
            if len(out) > cap:
                raise Bad("output")
            continue
        if kind == 1:
            lit = _code([8] * 144 + [9] * 112 + [7] * 24 + [8] * 8)
            dist = _code([5] * 30)
        else:
            hlit, hdist, hclen = take(5) + 257, take(5) + 1, take(4) + 4
            if hlit > 286 or hdist > 30:
                raise Bad("counts")
            cl = [0] * 19
            for k in range(hclen):
                cl[ORDER[k]] = take(3)
            table, lengths = _code(cl), []
            while len(lengths) < hlit + hdist:
                s = symbol(table)
                if s < 16:
                    lengths.append(s)
                elif s == 16:
                    if not lengths:
                        raise Bad("repeat")
                    lengths += [lengths[-1]] * (3 + take(2))
                else:
                    lengths += [0] * (3 + take(3) if s == 17 else 11 + take(7))
            if len(lengths) > hlit + hdist or not lengths[256]:
                raise Bad("lengths")
            lit, dist = _code(lengths[:hlit]), _code(lengths[hlit:])
        while True:
            s = symbol(lit)
            if s < 256:
                out.append(s)
            elif s == 256:
                break
            else:
                if s > 285:
                    raise Bad("length symbol")
                i = s - 257
                x = 0 if i < 8 or i == 28 else (i >> 2) - 1
                n = (3 + i if i < 8 else 258 if i == 28 else ((4 + (i & 3)) << x) + 3) + take(x)
                d = symbol(dist)
                if d > 29:
                    raise Bad("distance symbol")
                x = 0 if d < 4 else (d >> 1) - 1
                far = (d + 1 if d < 4 else ((2 + (d & 1)) << x) + 1) + take(x)
                if far > len(out):
                    raise Bad("distance")
                for _ in range(n):
                    out.append(out[-far])
            if len(out) > cap:
                raise Bad("output")
    return bytes(out)


def _compare(gpu, z, cap):
    try:
        want = plain_inflate(z, cap)
    except Bad:
        want = None
    try:
        got = gpu.decompress(z, gpu.Format.Raw, cap)
    except gpu.Error as e:
        assert e.code == -1
        got = None
    assert got == want
    return want


def test_plain_decoder_agrees_with_zlib(gpu):
    for kind in range(6):
        for level, strategy in ((6, 0), (9, zlib.Z_HUFFMAN_ONLY), (6, zlib.Z_FIXED), (0, 0)):
            d = synth.gen(5000, kind, kind)
            c = zlib.compressobj(level, zlib.DEFLATED, -15, 8, strategy)
            z = c.compress(d) + c.flush()
            assert plain_inflate(z, len(d)) == d
            _compare(gpu, z, len(d))
            assert _compare(gpu, z, len(d) - 1) is None


@pytest.mark.parametrize("seed", range(12))
def test_damaged_streams_against_a_plain_decoder(gpu, seed):
    r = random.Random(seed)
    rejected = 0
    for k in range(40):
        d = synth.gen(r.randrange(200, 6000), seed % 6, 100 * seed + k)
        c = zlib.compressobj(r.choice([1, 6, 9]), zlib.DEFLATED, -15, 8,
                             r.choice([0, 0, zlib.Z_HUFFMAN_ONLY, zlib.Z_RLE, zlib.Z_FIXED]))
        half = len(d) // 2
        z = bytearray(c.compress(d[:half]) + c.flush(r.choice([5, zlib.Z_SYNC_FLUSH, zlib.Z_NO_FLUSH])) + c.compress(d[half:]) + c.flush())
        if r.random() < 0.2:
            del z[r.randrange(1, len(z)):]
        for _ in range(r.randrange(1, 4)):
            # half of the damage in the first block's header
            z[r.randrange(min(len(z), 60 if r.random() < 0.5 else len(z)))] ^= 1 << r.randrange(8)
        want = _compare(gpu, bytes(z), 40000)
        rejected += want is None
    assert rejected


@pytest.mark.parametrize("n", [(68 << 20) + 12345, (33 << 20) + 1])
def test_outputs_larger_than_the_staging(gpu, n):
    d = synth.array(n, synth.MIXED, 3)
    z = zlib.compress(d.tobytes(), 1)
    assert np.array_equal(np.frombuffer(gpu.decompress(z, gpu.Format.Zlib, n + 5), np.uint8), d)
    m = (1 << 20) - 3
    z = b"".join(gzip.compress(d[o:o + m].tobytes(), 1, mtime=0) for o in range(0, n, m))
    assert np.array_equal(np.frombuffer(gpu.decompress(z, gpu.Format.Gzip, n), np.uint8), d)
