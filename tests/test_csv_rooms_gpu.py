"""CSV rows where the converter's way of taking them changes: windows sized for
short rows with rows around their edge among them, rows too long for any window
side by side, lines of many columns (written a lane a row), and bytes after a
field's closing quote."""

import random

import numpy as np
import pytest

from oracle import csv_map

pytestmark = pytest.mark.gpu


def convert(data):
    import torch
    import warpjq_b200 as wjq
    from warpjq_b200.shard import _DeviceBytes
    dev = torch.from_numpy(np.frombuffer(data, dtype=np.uint8).copy()).cuda()
    c = wjq.CsvConverter()
    d, n, used, rows = c.convert(dev.data_ptr(), len(data), stream=torch.cuda.current_stream().cuda_stream)
    assert used == len(data)
    out = bytes(torch.as_tensor(_DeviceBytes(d, max(1, n)), device="cuda").cpu().numpy()[:n])
    c.close()
    return out


def body(rng, n, kind):
    x = bytes(rng.choices(b"abcdefgh .:;", k=n))
    if kind == "quoted":
        x = b'"' + x.replace(b"e", b'""').replace(b".", b",").replace(b":", b"\n") + b'"'
    elif kind == "control":
        x = x.replace(b"a", b"\x01").replace(b"b", b"\t")
    return x


# the smallest window is 1,024 bytes, the largest 5,120 (8,192 for the lines)
@pytest.mark.parametrize("short, long", [(8, [990, 1000, 1005, 1008, 1009, 1010, 1020, 1024, 1100]), (8, [4000, 6000]),
                                         (100, [3900, 4080, 4096, 4100]), (300, [5090, 5104, 5105, 5119, 5121]),
                                         (2000, [1200, 1300, 7000]), (9000, [9000, 20]), (6000, [1270, 1275, 1280, 4000])])
@pytest.mark.parametrize("kind", ["plain", "quoted", "control"])
def test_rows_among_shorter_ones(short, long, kind):
    rng = random.Random(short + len(kind))
    rows = [b"a,b,c"]
    for i in range(400 if short < 1000 else 130):
        n = rng.choice(long) + rng.randrange(3) - 8 if rng.randrange(9) == 0 else max(1, short - 4)
        rows.append(b"%d,%s,%d" % (i, body(rng, n, kind), i % 7))
    data = b"\n".join(rows) + b"\n"
    assert convert(data) == csv_map.csv_to_ndjson(data)


@pytest.mark.parametrize("columns", [8, 9, 20, 60])
@pytest.mark.parametrize("width", [0, 1, 4, 7, 30, 90])
def test_many_columns(columns, width):
    rng = random.Random(columns * 100 + width)
    rows = [b",".join(b"name_%d" % k for k in range(columns))]
    for i in range(150):
        n = rng.randrange(columns + 2) if i % 5 == 0 else columns
        cell = lambda: rng.choice([b"%d" % rng.randrange(10**max(1, min(width, 9))), bytes(rng.choices(b"xy z", k=width)),
                                   b"", b'"' + b"q" * width + b'"', b'"a""b"' if width > 3 else b"7"])
        rows.append(b",".join(cell() for _ in range(n)))
    for end in (b"\n", b"\r\n"):
        data = end.join(rows)
        assert convert(data) == csv_map.csv_to_ndjson(data)


@pytest.mark.parametrize("pad", [0, 1, 2, 3, 40, 1500])
def test_bytes_after_a_closing_quote(pad):
    x = b"p" * pad
    tails = [b"z", b'"', b'y"y', b"\\", b"\x02", b"\t\t", b"q" * 50, b' "mid" ', b'""""'[:3], b"a\\b\"c\x01d"]
    rows = [b"a,b,c"]
    for t in tails:
        for inner in (b"", b"in", b'""', b"a,b", b"l\n", b"\\"):
            if (t.count(b'"') % 2):
                t = t + b'"'  # quotes stay even within a row
            rows += [b'%s"%s"%s,2,%s' % (b"", inner + x, t, x), b'1,"%s"%s' % (inner, t), b'"%s"%s,"%s"%s,3' % (inner, t, x, t)]
    data = b"\n".join(rows) + b"\n"
    assert convert(data) == csv_map.csv_to_ndjson(data)
