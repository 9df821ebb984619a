"""Levels 4-12, each input in a pass of its own: passes of few tiles take other
launch shapes (larger CTAs per tile) than the pass of all inputs, and emit the
same recorded streams; and a pass on both sides of the number of tiles at which
the shapes change."""
import hashlib
import json
import os
import zlib

import pytest

from lazy_inputs import cases
from orot_b200 import synth

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "lazy_streams.json")


@pytest.mark.parametrize("level", [4, 6, 9, 10, 12])
def test_one_input_per_pass(gpu, level):
    want = json.load(open(GOLDEN))[str(level)]
    bad = []
    for (name, d), w in zip(cases(), want):
        s = gpu.compress(d, level, gpu.Format.Raw)
        if hashlib.sha256(s).hexdigest()[:16] != w:
            bad.append(name)
    assert not bad


@pytest.mark.parametrize("level", [6, 10])
@pytest.mark.parametrize("kind", [synth.TEXT, synth.MIXED, synth.PERIODIC, synth.ZEROS])
def test_shapes_agree(gpu, level, kind):
    """The same 128 KiB blocks in passes of 1 to 1000 tiles."""
    block = 128 << 10
    data = synth.gen(30 * block, kind, 5)
    whole = gpu.ParallelCompressor(level, gpu.Format.Raw, 0, block).compress(data)
    assert zlib.decompress(whole, -15) == data
    for blocks in (1, 8, 9, 10, 18, 19):
        part = gpu.ParallelCompressor(level, gpu.Format.Raw, 0, block).compress(data[:blocks * block])
        # all but the last block, whose final bit and padding differ
        same = len(os.path.commonprefix([part, whole]))
        last = gpu.compress(data[(blocks - 1) * block:blocks * block], level, gpu.Format.Raw)
        assert same >= len(part) - len(last) - 16, blocks
        assert zlib.decompress(part, -15) == data[:blocks * block]
