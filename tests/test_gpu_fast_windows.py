"""Levels 1-3 at the edges of their 32-position windows: tiles of fewer windows
than warps that share a hash table, matches around the length that is measured
from preloaded words and around the longest, hashes that repeat inside a window
and runs that end at any place of one.  Byte parity with the oracle."""
import random

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu


def check(gpu, oracle, data, levels=(1, 2, 3)):
    b = gpu.DeviceBatch()
    for level in levels:
        b.load(b"".join(data), [len(d) for d in data], level, gpu.Format.Raw)
        b.run()
        for i, (d, n) in enumerate(zip(data, b.sizes())):
            assert b.output(i, n) == oracle.compress(d, level, 0), (level, i, len(d))
    b.close()


@pytest.mark.parametrize("tile", [32, 64, 96, 128, 160, 544])
def test_few_windows_per_tile(gpu, oracle, monkeypatch, tile):
    monkeypatch.setenv("OROT_B200_TILE", str(tile))
    sizes = [k * tile + e for k in (1, 2, 3, 5, 40) for e in (-1, 0, 1, 4)]
    check(gpu, oracle, [synth.gen(n, (0, 1, 2, 5)[i % 4], i) for i, n in enumerate(sizes)])


@pytest.mark.parametrize("tile", [0, 512])
def test_match_lengths(gpu, oracle, monkeypatch, tile):
    if tile:
        monkeypatch.setenv("OROT_B200_TILE", str(tile))
    r = random.Random(5)
    data = []
    for length in list(range(3, 36)) + [63, 64, 127, 128, 139, 140, 141, 255, 256, 257, 258, 259, 300, 517]:
        unit = bytes(r.randrange(256) for _ in range(length))
        d = bytearray()
        for k in range(24):  # at every offset from a window's start, distances of several sizes
            d += unit + bytes(r.randrange(256) for _ in range(1 + (k * 7) % 33))
        data.append(bytes(d))
        data.append(bytes(d) + unit)  # the match ends the data
    check(gpu, oracle, data)


@pytest.mark.parametrize("tile", [0, 96])
def test_repeats_inside_windows(gpu, oracle, monkeypatch, tile):
    if tile:
        monkeypatch.setenv("OROT_B200_TILE", str(tile))
    r = random.Random(6)
    data = []
    for period in (1, 2, 3, 4, 7, 15, 16, 31, 32, 33, 63):
        unit = bytes(r.randrange(256) for _ in range(period))
        for run in (33, 64, 95, 97, 400, 1000):
            d = bytes(r.randrange(256) for _ in range(r.randrange(70)))
            for _ in range(4):
                d += (unit * (run // period + 1))[:run] + bytes(r.randrange(4) for _ in range(r.randrange(1, 40)))
            data.append(d)
    # few byte values: several positions of a window share each hash
    data += [bytes(r.randrange(k) for _ in range(5000)) for k in (2, 3, 4)]
    # a candidate farther back than 32 KiB, and position 0 as the only candidate
    far = bytes(r.randrange(256) for _ in range(40))
    data += [far + bytes(r.randrange(256) for _ in range(n)) + far + far for n in (0, 32700, 32727, 32728, 32729, 70000)]
    check(gpu, oracle, data)
