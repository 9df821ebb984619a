"""Stored blocks around the sizes where the number of their pieces (65,535 bytes)
and of a piece's copies (4,096) changes, alone and beside coded blocks, against the oracle."""
import numpy as np
import pytest

from conftest import inflate
from orot_b200 import synth

pytestmark = pytest.mark.gpu
SIZES = [0, 1, 4095, 4096, 4097, 8192, 65534, 65535, 65536, 65535 + 4096, 65535 + 4097, 2 * 65535, 2 * 65535 + 1, 400000]


@pytest.mark.parametrize("level", [0, 1, 3, 6])
def test_batch_of_stored_and_coded_buffers(gpu, oracle, level):
    parts = []
    for i, n in enumerate(SIZES):
        parts += [synth.gen(n, 3, i) if n else b"", synth.gen(n, 0, i) if n else b""]  # random bytes, text
    b = gpu.DeviceBatch()
    b.load(np.frombuffer(b"".join(parts), np.uint8), [len(p) for p in parts], level, gpu.Format.Zlib)
    b.run()
    for i, (p, size) in enumerate(zip(parts, b.sizes())):
        got = b.output(i, size)
        assert inflate(got, 1) == p, (i, len(p))
        if level <= 3:
            assert got == oracle.compress(p, level, 1), (i, len(p))
    b.close()


@pytest.mark.parametrize("block", [4096, 4097, 65535, 65536, 70001])
@pytest.mark.parametrize("level", [0, 1, 6])
def test_chunks_stored_and_coded(gpu, oracle, level, block):
    d = b"".join(synth.gen(n, 3 if i % 2 else 0, i) for i, n in enumerate([block, block + 1, 3 * block - 5, 2 * block, 999]))
    cap = 2 * len(d) + 1024
    out = np.zeros(cap, np.uint8)
    ctx = gpu.ParallelCompressor(level, gpu.Format.Gzip, 0, block)
    n = gpu.lib().deflate_parallel_compress(ctx._ctx, np.frombuffer(d, np.uint8).ctypes.data, len(d), out.ctypes.data, cap)
    got = out[:n].tobytes()
    assert inflate(got, 2) == d
    if level <= 3:
        assert got == oracle.parallel(d, level, 2, block)
