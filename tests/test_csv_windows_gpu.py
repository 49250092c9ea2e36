"""CSV rows around the converter's staged windows (5,120 input and 8,192
output bytes a warp of 32 rows): rows that fill a window, exceed it alone or
with their neighbours, grow past the output's by escapes, and rows it hands on
(bytes after a closing quote) among ones it does not."""

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
    d, n, used, _ = c.convert(dev.data_ptr(), len(data), stream=torch.cuda.current_stream().cuda_stream)
    assert used == len(data)
    out = bytes(torch.as_tensor(_DeviceBytes(d, max(1, n)), device="cuda").cpu().numpy()[:n])
    c.close()
    return out


@pytest.mark.parametrize("size", [1, 15, 16, 150, 159, 160, 161, 1000, 5100, 5104, 5119, 5120, 5121, 9000])
@pytest.mark.parametrize("kind", ["plain", "quoted", "control", "odd", "mixed"])
def test_rows_around_the_windows(size, kind):
    rng = random.Random(size)
    rows = [b"a,b,c"]
    for i in range(70):
        n = max(0, size - 8 + rng.randrange(3))
        k = rng.choice(["plain", "quoted", "control", "odd", "number", "empty"]) if kind == "mixed" else kind
        if kind == "mixed" and rng.randrange(3):
            n = rng.randrange(60)
        body = bytes(rng.choice(b"abcdefgh .:;") for _ in range(n))
        if k == "quoted":
            body = b'"' + body.replace(b"e", b'""').replace(b"f", b"\\").replace(b".", b",").replace(b":", b"\n") + b'"'
        elif k == "control":
            body = body.replace(b"a", b"\x01").replace(b"b", b"\t")
        elif k == "odd":
            body = b'"' + body + b'"' + (b'x"y' if i % 2 else b"")
        elif k == "number":
            body = rng.choice([b"-0", b"1e5", b"12.50", b"01", b"1.", b"-", b"123456789012345678901"])
        elif k == "empty":
            body = b""
        rows.append(b"%d,%s,%s" % (i, body, rng.choice([b"", b"7", b"x"])) if k != "empty" or i % 2 else b"")
    for end in (b"\n", b"\r\n"):
        data = end.join(rows) + rng.choice([b"", end])
        assert convert(data) == csv_map.csv_to_ndjson(data), (size, kind, end)
