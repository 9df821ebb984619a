"""Workloads of the DEFLATE engine that are timed, each through a public entry point.

A case names its operation (`op`), the kind of data, sizes, level and format:

  call       deflate.compress of one bytes object, as a Python program calls it
  whole      deflate_compress (C ABI) of one buffer into the caller's buffer
  parallel   deflate_parallel_compress (C ABI): one stream in independent chunks
  resident   a device batch: buffers already on the GPU, one replay of its graph
             and every stream fetched into pinned memory
  batch      compress_pipelined: many buffers in one host-to-host call, pinned
  decode     deflate.decompress of one stream (compressed by zlib)
  members    deflate_decompress (C ABI) of a gzip file of independent members

Data kinds are the generators of orot_b200.synth: Zipf text, sorted 32-bit
integers, zeros, random bytes, a rotation of those four, and an 8-byte period
with 1% of the bytes replaced.
"""
import ctypes
import gzip
import math
import zlib

import numpy as np
import torch

from orot_b200 import deflate, synth

KINDS = {"text": synth.TEXT, "ints": synth.INTS, "zeros": synth.ZEROS, "random": synth.RANDOM,
         "mixed": synth.MIXED, "periodic": synth.PERIODIC}
FORMATS = {"raw": deflate.Format.Raw, "zlib": deflate.Format.Zlib, "gzip": deflate.Format.Gzip}

# Rough compressed fraction of each kind (fast levels, other levels), for work().
RATIO = {"text": (0.41, 0.28), "ints": (0.80, 0.55), "zeros": (0.012, 0.002), "random": (1.0, 1.0),
         "mixed": (0.60, 0.50), "periodic": (0.10, 0.04)}


def listed():
    return [
        # one small record or web response at the default level: latency only
        {"name": "call_4k_text_l6", "op": "call", "kind": "text", "bytes": 4096, "level": 6, "format": "zlib"},
        # a log block or column page at the fast level, ragged size
        {"name": "call_100k_ints_l1", "op": "call", "kind": "ints", "bytes": 100003, "level": 1, "format": "gzip"},
        # an ordinary object at the default level, ragged size
        {"name": "call_3m_mixed_l6", "op": "call", "kind": "mixed", "bytes": (3 << 20) + 17, "level": 6,
         "format": "zlib"},
        # the benchmark's single buffer: 16 MiB of text as one raw block
        {"name": "whole_16m_text_l1", "op": "whole", "kind": "text", "bytes": 16 << 20, "level": 1, "format": "raw"},
        # the benchmark's pigz-style file (a quarter of its size): 128 KiB chunks
        {"name": "parallel_64m_mixed_l6", "op": "parallel", "kind": "mixed", "bytes": 64 << 20, "level": 6,
         "format": "gzip", "block": 128 << 10},
        # archival at level 9 in 256 KiB chunks: text, and the input with the longest chains
        {"name": "parallel_32m_text_l9", "op": "parallel", "kind": "text", "bytes": 32 << 20, "level": 9,
         "format": "raw", "block": 256 << 10},
        {"name": "parallel_32m_periodic_l9", "op": "parallel", "kind": "periodic", "bytes": 32 << 20, "level": 9,
         "format": "raw", "block": 256 << 10},
        # the highest level, default chunk size
        {"name": "parallel_8m_mixed_l12", "op": "parallel", "kind": "mixed", "bytes": 8 << 20, "level": 12,
         "format": "zlib", "block": 0},
        # buffers of the headline batch (log-uniform 1 KiB to 4 MiB) kept on the GPU
        {"name": "resident_96_mixed_l1", "op": "resident", "kind": "mixed", "count": 96, "lo": 1 << 10,
         "hi": 4 << 20, "level": 1, "format": "zlib"},
        # a host-to-host batch of files at level 3
        {"name": "batch_48_mixed_l3", "op": "batch", "kind": "mixed", "count": 48, "lo": 64 << 10, "hi": 16 << 20,
         "level": 3, "format": "gzip"},
        # one ordinary stream decoded
        {"name": "decode_1m_text", "op": "decode", "kind": "text", "bytes": 1 << 20, "level": 6, "format": "zlib"},
        # a gzip file of 1 MiB members decoded at once
        {"name": "members_32m_mixed", "op": "members", "kind": "mixed", "bytes": 32 << 20, "level": 6,
         "member": 1 << 20},
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, uniform over its logarithm; mostly odd ones."""
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return max(lo, min(hi, n | 1 if rng.random() < 0.7 else n & ~15))


def draw(rng):
    op = rng.choice(["call", "call", "whole", "parallel", "parallel", "resident", "batch", "decode", "members"])
    kind = rng.choice(["text", "text", "mixed", "mixed", "ints", "zeros", "random", "periodic"])
    fmt = rng.choice(["raw", "zlib", "gzip"])
    level = rng.choice([1, 1, 2, 3, 4, 5, 6, 6, 6, 7, 9, 9, 12])
    case = {"op": op, "kind": kind, "level": level, "format": fmt}
    if op == "call":
        case["bytes"] = _log(rng, 1 << 10, 4 << 20)
    elif op == "whole":
        case["bytes"] = _log(rng, 1 << 20, 16 << 20)
    elif op == "parallel":
        case["bytes"] = _log(rng, 1 << 20, 8 << 20 if level > 9 else 32 << 20 if level > 6 else 64 << 20)
        case["block"] = rng.choice([0, 64 << 10, 128 << 10, 256 << 10, 100001])
    elif op == "resident":
        case["count"] = rng.randint(8, 96)
        case["lo"], case["hi"] = 1 << 10, _log(rng, 64 << 10, 4 << 20 if level <= 6 else 1 << 20)
    elif op == "batch":
        case["count"] = rng.randint(8, 48)
        case["lo"], case["hi"] = 4 << 10, _log(rng, 1 << 20, 16 << 20 if level <= 3 else 4 << 20)
        if level > 9:
            case["hi"] = 1 << 20
    elif op == "decode":
        case["bytes"] = _log(rng, 1 << 10, 1 << 20)
        case["level"] = rng.choice([1, 6, 6, 9])
    else:
        case["bytes"] = _log(rng, 4 << 20, 32 << 20)
        case["level"] = rng.choice([1, 6, 6, 9])
        case["member"] = rng.choice([256 << 10, 1 << 20, 333333])
        del case["format"]
    return case


def _synth(out, kind, seed):
    synth.fill(out, kind, seed)
    if kind == synth.ZEROS:  # zero fill behind a short header, as in a sparse file
        out[:16] = synth.array(16, synth.RANDOM, seed)[:out.size]
    return out


def _data(case, seed):
    return _synth(np.empty(case["bytes"], np.uint8), KINDS[case["kind"]], seed)


def _sizes(case):
    """The buffer sizes belong to the case; the seed makes the bytes."""
    return synth.loguniform_sizes(case["count"], case["lo"], case["hi"], case["hi"])


def _fill_buffers(case, sizes, seed, out):
    """Buffers back to back; those of a mixed batch take the four plain kinds in turn."""
    o = 0
    for i, n in enumerate(int(x) for x in sizes):
        kind = i % 4 if case["kind"] == "mixed" else KINDS[case["kind"]]
        _synth(out[o:o + n], kind, seed * 1000003 + i)
        o += n


def _pinned(n):
    return torch.zeros(max(int(n), 1), dtype=torch.uint8, pin_memory=True).numpy()


def _deflated(data, level, fmt):
    c = zlib.compressobj(level, zlib.DEFLATED, {"raw": -15, "zlib": 15, "gzip": 31}[fmt])
    return c.compress(data) + c.flush()


def prepare(case, seed):
    op = case["op"]
    s = {"op": op, "level": case["level"], "fmt": FORMATS[case.get("format", "gzip")]}
    if op == "call":
        s["data"] = _data(case, seed).tobytes()
        s["out"] = np.zeros(deflate.compress_bound(case["bytes"], s["fmt"]), np.uint8)
    elif op in ("whole", "parallel"):
        s["data"] = _data(case, seed)
        n, extra = case["bytes"], 0
        if op == "parallel":
            block = case["block"]
            s["ctx"] = deflate.ParallelCompressor(case["level"], s["fmt"], 0, block)
            extra = 16 * (n // (block or (128 << 10)) + 2)
        s["out"] = np.zeros(deflate.compress_bound(n, s["fmt"]) + extra, np.uint8)
    elif op == "resident":
        sizes = _sizes(case)
        concat = np.empty(int(sizes.sum()), np.uint8)
        _fill_buffers(case, sizes, seed, concat)
        s["batch"] = deflate.DeviceBatch()
        s["batch"].load(concat, [int(x) for x in sizes], case["level"], s["fmt"])
        caps = [deflate.compress_bound(int(x), s["fmt"]) for x in sizes]
        s["slots"] = np.concatenate([[0], np.cumsum(caps)]).tolist()
        s["out"] = _pinned(s["slots"][-1])
    elif op == "batch":
        s["sizes"] = _sizes(case)
        s["data"] = _pinned(s["sizes"].sum())
        _fill_buffers(case, s["sizes"], seed, s["data"])
        s["out"] = _pinned(deflate.packed_bound([int(x) for x in s["sizes"]], s["fmt"]))
    elif op == "decode":
        s["n"] = case["bytes"]
        s["data"] = _deflated(_data(case, seed).tobytes(), case["level"], case["format"])
    else:
        plain, m = _data(case, seed).tobytes(), case["member"]
        packed = b"".join(gzip.compress(plain[o:o + m], case["level"], mtime=0) for o in range(0, len(plain), m))
        s["data"] = np.frombuffer(packed, np.uint8)
        s["out"] = np.zeros(case["bytes"], np.uint8)
    return s


def run(s):
    """Compressed sizes come with the whole output buffer (zero past the last byte written)."""
    op, level, fmt = s["op"], s["level"], s["fmt"]
    L = deflate.lib()
    if op == "call":
        got = deflate.compress(s["data"], level, fmt)
        s["out"][:len(got)] = np.frombuffer(got, np.uint8)  # the caller's page or record
        return [len(got), s["out"]]
    if op == "whole":
        n = L.deflate_compress(s["data"].ctypes.data, s["data"].size, s["out"].ctypes.data, s["out"].size, level,
                               int(fmt))
        return [n, s["out"]]
    if op == "parallel":
        n = L.deflate_parallel_compress(s["ctx"]._ctx, s["data"].ctypes.data, s["data"].size, s["out"].ctypes.data,
                                        s["out"].size)
        return [n, s["out"]]
    if op == "resident":
        b, slots, out = s["batch"], s["slots"], s["out"].ctypes.data
        b.run(graph=True)
        sizes = b.sizes()
        for i, n in enumerate(sizes):
            L.deflate_gpu_batch_output(b._b, i, out + slots[i], n)
        return [np.array(sizes), s["out"]]
    if op == "batch":
        _, offs, sizes = deflate.compress_pipelined(s["data"], s["sizes"], level, fmt, s["out"])
        return [offs.view(np.int64), sizes.view(np.int64), s["out"]]
    if op == "decode":
        return np.frombuffer(deflate.decompress(s["data"], fmt, s["n"]), np.uint8)
    got = ctypes.c_size_t(0)
    L.deflate_decompress(s["data"].ctypes.data, s["data"].size, s["out"].ctypes.data, s["out"].size,
                         ctypes.byref(got), int(fmt))
    return s["out"][:got.value]


def work(case):
    """Each input byte read once and each output byte written once."""
    if case["op"] in ("resident", "batch"):
        plain = int(_sizes(case).sum())
    else:
        plain = case["bytes"]
    return {"bytes": plain * (1 + RATIO[case["kind"]][0 if case["level"] <= 3 else 1]), "flops": 0}


def exact(case, seed):
    """A decoder returns the bytes that were compressed; a compressor's stream has no other form to hold it to."""
    return _data(case, seed) if case["op"] in ("decode", "members") else None
