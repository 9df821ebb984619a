"""The tuner's candidates are what its table entries mean: values in place of a
row of the geometry table, through one environment switch."""
import hashlib
import os
import re

import pytest

from orot_b200 import synth, tune

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))


def _rows(path):
    return [(int(m.group(1)) << int(m.group(2) or 0), [int(x) for x in m.groups()[2:]]) for m in
            re.finditer(r"\{(\d+)ull(?: << (\d+))?, (\d+), (\d+), \{(\d+), (\d+), (\d+)\}\}", open(path).read())]


def test_classes_are_the_rows_of_the_table():
    rows = _rows(tune.TABLE)
    assert [lo for lo, _ in rows] == tune.CLASSES
    assert len(tune.CLASS_BYTES) == len(tune.CLASSES)
    for i, n in enumerate(tune.CLASS_BYTES):  # each class is timed at a size of its own
        assert n >= tune.CLASSES[i] and (i + 1 == len(tune.CLASSES) or n < tune.CLASSES[i + 1])


def test_a_candidate_sets_one_entry_of_the_row():
    assert tune.row_with(0, 4096) == "4096,65536,32"
    assert tune.row_with(1, 8192) == "65536,8192,32"
    assert tune.row_with(2, 4) == "65536,65536,4"


def test_the_smallest_of_equal_candidates_is_kept():
    assert tune.pick([(1.00, 65536), (1.01, 4096), (1.05, 1024)]) == (1.01, 4096)
    assert tune.pick([(2.0, 1), (1.0, 2), (1.5, 4)]) == (1.0, 2)


def test_a_written_table_holds_the_rows(tmp_path):
    rows = [{"min_bytes": lo, "tile12": 4096 << (i % 3), "tile14": 8192, "run": [i + 1, 9, 32]} for i, lo in enumerate(tune.CLASSES)]
    out = str(tmp_path / "geometry_table.h")
    tune.write_table(rows, "a test", out)
    assert _rows(out) == [(r["min_bytes"], [r["tile12"], r["tile14"], *r["run"]]) for r in rows]


@pytest.mark.gpu
def test_the_row_does_not_change_the_output(gpu, monkeypatch):
    sizes = [3000000, 70000, 1, 12000]
    data = b"".join(synth.gen(n, synth.MIXED if i == 0 else i, i) for i, n in enumerate(sizes))
    for level in (1, 3, 6, 12):
        seen = set()
        for row in (None, "512,512,1", "65536,65536,32", "1024,4096,5", "not a row"):
            if row is None:
                monkeypatch.delenv("OROT_B200_GEOMETRY", raising=False)
            else:
                monkeypatch.setenv("OROT_B200_GEOMETRY", row)
            b = gpu.DeviceBatch()
            b.load(data, sizes, level, gpu.Format.Gzip)
            b.run()
            seen.add(hashlib.sha256(b"".join(b.output(i, n) for i, n in enumerate(b.sizes()))).hexdigest())
            b.close()
        assert len(seen) == 1, level


@pytest.mark.gpu
def test_the_row_limits_tiles(gpu, monkeypatch):
    """A row's tile limits what the planner takes (device memory: one table per tile)."""
    import torch
    torch.cuda.init()
    used = {}
    for row in ("512,512,32", "4096,4096,32", "65536,65536,32"):
        monkeypatch.setenv("OROT_B200_GEOMETRY", row)
        b = gpu.DeviceBatch()
        free = torch.cuda.mem_get_info()[0]
        b.load(bytes(8 << 20), [8 << 20], 3, gpu.Format.Raw)
        used[row] = free - torch.cuda.mem_get_info()[0]
        b.close()
    # 16,384, 2,048 and (cut finer than the limit) 1,024 tables of 64 KiB
    assert used["512,512,32"] > 1 << 30 > used["4096,4096,32"] > 128 << 20 > used["65536,65536,32"] > 64 << 20
