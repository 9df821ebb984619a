"""What the server charges to its device budget for a request is what the
planner lays out for it, tables of small tiles included."""
import numpy as np
import pytest

from orot_b200 import deflate, synth

MIB = 1 << 20


@pytest.mark.parametrize("level, bits", [(1, 12), (3, 14)])
def test_tables_of_small_tiles_are_charged(level, bits):
    for n in (100000, 380 << 10, MIB, 3 * MIB, 20 * MIB):
        tile = deflate.geometry_tile(n, 148, bits)
        tables = ((n + tile - 1) // tile - 1) * (4 << bits)
        need = deflate.device_bytes(n, n, level)
        assert tables + 7 * n <= need <= 1.1 * tables + 11 * n, n
        # in a large pass the same stream has fewer tiles
        assert deflate.device_bytes(n, 256 * MIB, level) <= 11 * n
    assert deflate.device_bytes(380 << 10, 380 << 10, 3) > 50e6


@pytest.mark.parametrize("level", [0, 4, 6, 9, 12])
def test_other_levels_do_not_depend_on_the_pass(level):
    for n in (1, 1000, 70000, 5 * MIB):
        need = deflate.device_bytes(n, n, level)
        assert need == deflate.device_bytes(n, 256 * MIB, level)
        assert (3 if level == 0 else 9) * n <= need <= (3.1 if level == 0 else 9.3) * n + 8192


@pytest.mark.gpu
@pytest.mark.parametrize("level", [0, 1, 3, 6])
@pytest.mark.parametrize("n", [1000003, 9 * MIB + 1, 40 * MIB])
def test_charge_covers_what_a_pass_allocates(gpu, level, n):
    import torch
    torch.cuda.init()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    b = gpu.DeviceBatch()
    data = np.zeros(n, np.uint8)
    free = torch.cuda.mem_get_info()[0]
    b.load(data, [n], level, gpu.Format.Gzip)
    used = free - torch.cuda.mem_get_info()[0]
    b.close()
    charged = gpu.device_bytes(n, n, level, sms)
    packed = gpu.compress_bound(n, gpu.Format.Gzip)  # a batch that is only loaded has no packed output
    assert used <= charged + 8 * MIB  # four arenas, each rounded up
    assert charged - packed <= 1.05 * used + 8 * MIB


@pytest.mark.gpu
def test_a_small_budget_serves_all(gpu):
    data = [synth.gen(380 << 10, i % 4, i) for i in range(12)]
    srv = gpu.Server(device_budget=64 << 20, lanes=2)
    tickets = [srv.submit(d, 3, gpu.Format.Zlib) for d in data]
    for t, d in zip(tickets, data):
        assert srv.wait(t, timeout=120)[0] == gpu.compress(d, 3, gpu.Format.Zlib)
    srv.close()
