"""Levels 4-12 emit a fixed stream: the matches are those of the documented
search (newest first, chain, skip and miss limits, nice length) whatever the
grouping of tiles.  The digests in golden/lazy_streams.json were recorded from
the one-CTA-per-run search that walked every chain step by step; every byte
must stay as it was, for every grouping, and inflate to the input."""
import hashlib
import json
import os
import zlib

import pytest

from lazy_inputs import cases

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "lazy_streams.json")


def digest(streams) -> str:
    h = hashlib.sha256()
    for s in streams:
        h.update(len(s).to_bytes(8, "little") + s)
    return h.hexdigest()


def compress_all(gpu, level):
    data = [d for _, d in cases()]
    b = gpu.DeviceBatch()
    b.load(b"".join(data), [len(d) for d in data], level, gpu.Format.Raw)
    b.run()
    out = [b.output(i, n) for i, n in enumerate(b.sizes())]
    b.close()
    return data, out


@pytest.mark.parametrize("level", range(4, 13))
def test_streams_are_as_recorded(gpu, level):
    data, out = compress_all(gpu, level)
    for d, s in zip(data, out):
        assert zlib.decompress(s, -15) == d
    want = json.load(open(GOLDEN))[str(level)]
    got = [hashlib.sha256(s).hexdigest()[:16] for s in out]
    bad = [name for (name, _), g, w in zip(cases(), got, want) if g != w]
    assert not bad and len(got) == len(want)


@pytest.mark.parametrize("run", [1, 2, 9, 32])
def test_grouping_does_not_matter(gpu, monkeypatch, run):
    for level in (4, 9, 10):
        monkeypatch.delenv("OROT_B200_LAZY_RUN", raising=False)
        want = digest(compress_all(gpu, level)[1])
        monkeypatch.setenv("OROT_B200_LAZY_RUN", str(run))
        assert digest(compress_all(gpu, level)[1]) == want
