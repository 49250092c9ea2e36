"""Rows of values around the lengths where their copy changes hands: a thread's
own rows, rows of a group of lanes beside them in one staged batch, batches too
large to stage, and the same rows printed by a mixed batch."""

import random

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu

QUERIES = [".v", "{a: .v, b: .none, c: .w}", "select(.n < 3) | .v"]
SIZES = {"short": [0, 1, 2, 3, 4, 5, 20], "own": [124, 125, 126, 127, 128], "mid": [60, 61, 62, 63, 64, 65],
         "long": [8180, 8188, 8189, 8190, 8193, 20000], "mixed": [0, 5, 30, 30, 30, 30, 127, 300, 4000],
         "rare": [10] * 200 + [7000]}


def lines(sizes, n, seed):
    rng = random.Random(seed)
    out = []
    for i in range(n):
        k = rng.choice(sizes)
        v = bytes(rng.choices(b"abcdefgh ,;0123456789", k=k))
        v = b'"%s"' % v if rng.randrange(8) else rng.choice([b"null", b"true", b"-1.5e3", b'"a\\"b\\u0041"', b"[1,2]"])
        out.append(b'{"n":%d,"v":%s%s}' % (rng.randrange(5), v, b',"w":%d' % i if rng.randrange(4) else b""))
    return b"\n".join(out) + b"\n"


def take(ptr, n):
    import torch
    from warpjq_b200.shard import _DeviceBytes
    return bytes(torch.as_tensor(_DeviceBytes(ptr, max(1, n)), device="cuda").cpu().numpy()[:n])


@pytest.mark.parametrize("fmt", ["ndjson", "csv"])
@pytest.mark.parametrize("kind", list(SIZES))
def test_value_rows(kind, fmt):
    import torch
    import warpjq_b200 as wjq
    data = lines(SIZES[kind], 300 if kind == "long" else 1500, len(kind))
    stream = torch.cuda.current_stream().cuda_stream
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    head = {q: 0 for q in QUERIES}
    for query in QUERIES:
        want = orc.run(query, data, fmt=fmt).out
        if fmt == "csv":
            head[query] = want.index(b"\n") + 1
        q = wjq.Query(query, fmt, chunk_bytes=1 << 20)
        q.launch_device(dev.data_ptr(), len(data), stream)
        r = q.collect_device()
        got = take(r.d_out_bytes, r.out_len)
        assert got == want[head[query]:], (kind, query)
        off = np.frombuffer(take(r.d_out_row_off, 8 * (r.n_selected + 1)), dtype=np.int64)
        ends = [i + 1 for i, c in enumerate(got) if c == 10]  # no row holds a newline here
        assert list(off) == [0] + ends
        q.close()
    # three queries over the parts of one batch
    cut = data.index(b"\n", len(data) // 2) + 1
    parts = [data[:cut], data[cut:], data[:cut]]
    offs, total = [], 0
    for p in parts:
        total = (total + 15) & ~15
        offs.append(total)
        total += len(p)
    host = np.zeros(total + 16, dtype=np.uint8)
    for p, o in zip(parts, offs):
        host[o:o + len(p)] = np.frombuffer(p, dtype=np.uint8)
    dev = torch.from_numpy(host).cuda()
    qs = [wjq.Query(x, fmt, chunk_bytes=1 << 20) for x in QUERIES]
    qs[0].batch_launch_mixed(qs, dev.data_ptr(), offs, [len(p) for p in parts], stream)
    items, every = qs[0].batch_collect()
    got = wjq.batch_outputs_mixed(qs, items, every, host)
    assert got == [orc.run(x, p, fmt=fmt).out for x, p in zip(QUERIES, parts)]
    for q in qs:
        q.close()
