"""Planning of a stream's blocks: stored blocks (whose padding depends on the bit
they start at) among coded ones at every place of a group of 32, in streams on
both sides of the number of segments that is planned by a CTA per segment, and
segments of more tiles than a CTA has threads.  Byte parity with the oracle."""
import random

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu
BLOCK = 32768


@pytest.mark.parametrize("segments", [1, 31, 32, 33, 64, 97, 1024, 1025])
def test_stored_among_coded(gpu, oracle, segments):
    r = random.Random(segments)
    parts = [synth.gen(BLOCK, synth.RANDOM if r.random() < 0.4 else synth.TEXT, k) for k in range(min(segments, 64))]
    data = b"".join(parts[k % len(parts)] for k in r.choices(range(len(parts)), k=segments - 1)) + parts[0][:BLOCK - 7]
    for fmt in (0, 2):
        assert gpu.ParallelCompressor(1, gpu.Format(fmt), 0, BLOCK).compress(data) == oracle.parallel(data, 1, fmt, BLOCK)
    out = gpu.ParallelCompressor(6, gpu.Format.Raw, 0, BLOCK).compress(data)
    assert gpu.decompress(out, gpu.Format.Raw, len(data)) == data


@pytest.mark.parametrize("tiles", [255, 256, 257, 600])
@pytest.mark.parametrize("kind", [synth.TEXT, synth.RANDOM, synth.ZEROS])
def test_many_tiles_per_segment(gpu, oracle, monkeypatch, tiles, kind):
    monkeypatch.setenv("OROT_B200_TILE", "512")
    data = synth.gen(tiles * 512 - 3, kind, tiles)
    b = gpu.DeviceBatch()
    for level in (1, 2):
        b.load(data, [len(data)], level, gpu.Format.Zlib)
        b.run()
        assert b.output(0, b.sizes()[0]) == oracle.compress(data, level, 1)
    b.close()
