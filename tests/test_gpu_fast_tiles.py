"""Levels 1-3 cut into tiles: hash tables carried in chunks of 32 tiles, and
runs that cross whole tiles (their parses of different phase never meet, so the
tiles' entries follow by arithmetic).  Byte parity with the oracle for every
tile size, at the edges of tiles, chunks and runs; and stored blocks, whose
copies are cut into parts of 4 KiB."""
import random

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu
TILES = [512, 1024, 4096]


def check(gpu, oracle, data, levels=(1, 2, 3)):
    b = gpu.DeviceBatch()
    for level in levels:
        b.load(b"".join(data), [len(d) for d in data], level, gpu.Format.Zlib)
        b.run()
        for i, (d, n) in enumerate(zip(data, b.sizes())):
            assert b.output(i, n) == oracle.compress(d, level, 1), (level, i, len(d))
    b.close()


@pytest.mark.parametrize("tile", TILES)
def test_chunks_of_tiles(gpu, oracle, monkeypatch, tile):
    monkeypatch.setenv("OROT_B200_TILE", str(tile))
    sizes = [k * tile + e for k in (1, 2, 32, 33, 34, 64, 65, 66, 100) for e in (-1, 0, 1)]
    check(gpu, oracle, [synth.gen(n, i % 2, i) for i, n in enumerate(sizes)])


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("period", [1, 2, 3, 8, 31, 32, 33, 300])
def test_runs_across_tiles(gpu, oracle, monkeypatch, tile, period):
    monkeypatch.setenv("OROT_B200_TILE", str(tile))
    r = random.Random(period)
    unit = bytes(r.randrange(256) for _ in range(period))
    data = []
    for lead in (0, 1, 100, tile - 1, tile, 3 * tile + 7):
        for run in (tile + 257, 2 * tile + 288, 5 * tile, 5 * tile + 31, 40 * tile + 259):
            head = synth.gen(lead, synth.TEXT, run)
            data.append(head + (unit * (run // period + 1))[:run] + synth.gen(r.randrange(700), synth.TEXT, lead))
    # a run whose bytes change once, at and around tile edges
    for at in (8 * tile - 2, 8 * tile - 1, 8 * tile, 8 * tile + 1, 8 * tile + 257, 9 * tile - 33):
        d = bytearray((unit * (20 * tile // period + 1))[:20 * tile])
        d[at] ^= 0x55
        data.append(bytes(d))
    check(gpu, oracle, data, (1, 3))


def test_small_passes_and_stored_blocks(gpu, oracle):
    """The tile sizes the planner picks itself."""
    for n in (1, 511, 512, 513, 4096, 65535, 65536, 131071, 300000, 1 << 20, (3 << 20) + 5):
        for kind in (synth.MIXED if n > (1 << 20) else synth.TEXT, synth.RANDOM, synth.ZEROS):
            d = synth.gen(n, kind, n)
            for level, fmt in ((0, 2), (1, 0), (3, 2)):
                assert gpu.compress(d, level, gpu.Format(fmt)) == oracle.compress(d, level, fmt), (n, kind, level)
    d = synth.gen(1 << 20, synth.RANDOM, 3)
    for block in (32768, 65535, 65537, 131072):
        for level in (1, 6):
            out = gpu.ParallelCompressor(level, gpu.Format.Raw, 0, block).compress(d)
            if level == 1:
                assert out == oracle.parallel(d, level, 0, block)
            assert gpu.decompress(out, gpu.Format.Raw, len(d)) == d
