"""orot_b200_geometry_tile answers with the tile the planner cuts a pass into,
which is finer than the table's below a few MiB (no GPU needed)."""
import pytest

from orot_b200 import deflate

MIB = 1 << 20


@pytest.mark.parametrize("bits, sizes", [
    (12, [(1, 512), (100003, 512), (MIB - 512, 512), (MIB - 511, 1024), (MIB, 1024), (2 * MIB - 1024, 1024),
          (2 * MIB - 1023, 2048), (8 * MIB - 2048, 2048), (8 * MIB - 2047, 4096), (8 * MIB, 4096), (64 * MIB, 16384)]),
    (14, [(1, 512), (767 * 512, 512), (767 * 512 + 1, 1024), (767 * 1024, 1024), (767 * 1024 + 1, 2048),
          (767 * 2048, 2048), (767 * 2048 + 1, 4096), (8 * MIB - 1, 4096), (8 * MIB, 8192)]),
])
def test_small_passes_are_cut_finer(bits, sizes):
    for n, tile in sizes:
        assert deflate.geometry_tile(n, 148, bits) == tile, n
        # the same work per SM
        assert deflate.geometry_tile(2 * n, 296, bits) == tile, n


@pytest.mark.parametrize("bits", [12, 14])
def test_tiles_grow_with_the_pass(bits):
    last = 0
    for k in range(200):
        t = deflate.geometry_tile(int(2 ** (k / 6)) + 1, 148, bits)
        assert t >= last and t & (t - 1) == 0 and 512 <= t <= 65536
        last = t
