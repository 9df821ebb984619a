"""gzip files of several members decoded one after the other (files below 256 KiB,
and longer ones whose members cannot be told apart by scanning): a member's output
begins where the one before ended, at any byte."""
import gzip

import pytest

from orot_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1000, 2000], [1, 1, 1, 70000], [16, 32, 48], [7, 65535, 65537, 3], [100001, 99999, 0, 5],
                                   [4097] * 9])
def test_members_of_any_size(gpu, sizes):
    for kind in (0, 3):
        parts = [synth.gen(n, kind, 10 * n + i) if n else b"" for i, n in enumerate(sizes)]
        packed = [gzip.compress(p, 6, mtime=0) for p in parts]
        data, file = b"".join(parts), b"".join(packed)
        assert gpu.decompress(file, gpu.Format.Gzip, len(data)) == data
        for k in range(len(packed)):  # a wrong checksum fails, whichever member has it
            bad = bytearray(packed[k])
            bad[-8] ^= 1
            with pytest.raises(gpu.Error) as e:
                gpu.decompress(b"".join(packed[:k] + [bytes(bad)] + packed[k + 1:]), gpu.Format.Gzip, len(data))
            assert e.value.code == -1
        assert gpu.decompress(file, gpu.Format.Gzip, len(data)) == data


def test_a_member_that_looks_like_two(gpu):
    """A stored member of 300,000 bytes whose data holds a gzip header: the scan splits it there."""
    d = bytearray(synth.gen(300000, 3, 5))
    d[150001:150011] = bytes([0x1F, 0x8B, 8, 0, 0, 0, 0, 0, 0, 3])
    parts = [synth.gen(777, 0, 1), bytes(d), synth.gen(12345, 1, 2)]
    file = b"".join(gzip.compress(p, 1, mtime=0) for p in parts)
    data = b"".join(parts)
    assert bytes(d[150001:150011]) in file and gzip.decompress(file) == data
    assert gpu.decompress(file, gpu.Format.Gzip, len(data)) == data
