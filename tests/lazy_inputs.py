"""Inputs for the exact-output tests of levels 4-12: sizes around the tile, the
search group and the window, and data that meets every end of a chain walk."""
import random

from orot_b200 import synth

TILE, WINDOW = 16 * 258, 32768
SIZES = [1, 3, 4, 5, 31, 33, TILE - 1, TILE, TILE + 1, TILE + 64, 2 * TILE + 97, 9 * TILE, 9 * TILE + 3,
         WINDOW + 3, WINDOW + TILE - 2, 20 * TILE + 17, 300007]


def colliding_words(n: int, seed: int) -> bytes:
    """4-byte words of one 15-bit hash bucket, of both its 16-bit hashes, in
    random order with a few other bytes between: walks full of skipped
    candidates, of misses, and of budgets that run out."""
    inv = pow(0x9E3779B1, -1, 1 << 32)  # v = h * inv has the hash h >> 17
    r = random.Random(seed)
    words = [((0x1234 << 17 | half << 16 | r.randrange(1 << 16)) * inv & 0xFFFFFFFF).to_bytes(4, "little")
             for half in (0, 1) for _ in range(12)]
    out = bytearray()
    while len(out) < n:
        out += r.choice(words)
        if r.random() < 0.3:
            out += bytes(r.choices(b"ab", k=r.randrange(3)))
    return bytes(out[:n])


def two_chains(n: int, seed: int) -> bytes:
    """Long stretches of one 16-bit hash after another in the same bucket: the
    budget of skipped candidates ends the walk."""
    inv = pow(0x9E3779B1, -1, 1 << 32)
    a, b = (((0x2BCD << 17 | half << 16 | 0x1357) * inv & 0xFFFFFFFF).to_bytes(4, "little") for half in (0, 1))
    r = random.Random(seed)
    out = bytearray()
    while len(out) < n:
        w = a if r.random() < 0.5 else b
        for _ in range(r.randrange(1, 600)):
            out += w + bytes([r.randrange(4)])
    return bytes(out[:n])


def fibonacci(symbols: int) -> bytes:
    """Shuffled bytes whose counts are the Fibonacci numbers: the deepest tree."""
    counts = [1, 1]
    while len(counts) < symbols:
        counts.append(counts[-1] + counts[-2])
    body = bytearray(b"".join(bytes([i * 7 & 255]) * c for i, c in enumerate(counts)))
    random.Random(symbols).shuffle(body)
    return bytes(body)


def cases():
    """(name, data) in a fixed order; data is deterministic."""
    for kind in range(6):
        for n in SIZES:
            if n > TILE or kind in (0, 2):
                yield f"{kind}:{n}", synth.gen(n, kind, 100 + kind)
    for name, make in (("collide", colliding_words), ("chains", two_chains)):
        for n in (TILE + 5, 120001):
            yield f"{name}:{n}", make(n, n)
    for n in (18, 22, 25):  # code lengths beyond 15 bits without a limit
        yield f"fibonacci:{n}", fibonacci(n)
    yield "every byte once", bytes(range(256))
    yield "every byte, few often", bytes(range(256)) + bytes(random.Random(2).choices(b"abcd", k=30000))
    text = synth.gen(50000, synth.TEXT, 5)
    yield "text+zeros+text", text + bytes(40000) + text
    yield "rare tail", b"".join(bytes([i & 255, 1, 2, 3, 4, 5, 6, i >> 8]) for i in range(9000))
