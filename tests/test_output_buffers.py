"""Buffers the library writes into have to be writable: an immutable object is
refused before anything is written (no GPU needed)."""
import ctypes

import numpy as np
import pytest

from orot_b200 import deflate


def _read_only():
    frozen = np.zeros(4096, np.uint8)
    frozen.flags.writeable = False
    return [bytes(4096), memoryview(bytes(4096)), memoryview(bytearray(4096)).toreadonly(), frozen,
            np.frombuffer(bytes(4096), np.uint8), np.zeros((64, 128), np.uint8)[:, ::2]]


@pytest.mark.parametrize("k", range(6))
@pytest.mark.parametrize("call", [deflate.compress_packed, deflate.compress_pipelined])
def test_read_only_outputs_are_refused(k, call):
    out = _read_only()[k]
    with pytest.raises(TypeError):
        call(b"a" * 100, [100], 6, deflate.Format.Zlib, out)
    assert not any(bytes(out) if k != 5 else out.tobytes())


def test_writable_outputs_are_addressed_in_place():
    a = np.zeros((3, 50), np.uint16)
    for out, n in ((bytearray(77), 77), (ctypes.create_string_buffer(33), 33), (a, 300), (memoryview(bytearray(20)), 20)):
        addr, size, keep = deflate._outptr(out)
        assert size == n
        ctypes.memset(addr, 0x5A, n)
        assert bytes(memoryview(out).cast("B")) == b"Z" * n
        del keep


@pytest.mark.gpu
def test_server_refuses_a_read_only_output(gpu):
    srv = gpu.Server(lanes=1)
    with pytest.raises(TypeError):
        srv.submit(b"a" * 100, 6, gpu.Format.Zlib, out=bytes(4096))
    out = bytearray(4096)
    got, _ = srv.wait(srv.submit(b"a" * 100, 6, gpu.Format.Zlib, out=out), timeout=60)
    assert got == gpu.compress(b"a" * 100, 6, gpu.Format.Zlib) == bytes(out[:len(got)])
    srv.close()
