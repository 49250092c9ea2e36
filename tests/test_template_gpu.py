"""Lines that fit the run's line template beside lines that do not, in one
round of a warp, over inputs with enough tiles for templates to be made and
used: the mixture from which a template is given up included, alone and with a
template per query in a mixed batch."""

import random

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu

QUERIES = ["select(.status == 500) | count", "select(.status >= 500) | {p: .path, b: .bytes}",
           "group_by(.host) | sum(.bytes)", ".ua", "select(.latency_ms > 50) | .method", "avg(.latency_ms)"]
# lines per 1,000 that are not of the common shape
RATES = [1, 20, 300]


def lines(n_bytes, rate, seed):
    import warpjq_b200 as wjq
    rng = random.Random(seed)
    buf, used, _ = wjq.gen_nginx(n_bytes, seed=seed)
    out = bytes(buf[:used]).split(b"\n")[:-1]
    for i in range(len(out)):
        x = out[i]
        if rng.randrange(1000) >= rate:
            continue
        out[i] = rng.choice([
            x + b"\r", x.replace(b'":', b'" : ', 1), x.replace(b',"', b', "'), x[:-1] + b',"tags":[1,"a"]}',
            x[:rng.randrange(len(x))], x.replace(b'"status":', b'"status":0'), x[:-1], x + b"}", b"", b" \t ", b"5",
            x.replace(b'"path":"', b'"path":"\\u00e9\\"'), x.replace(b'"path":"', b'"path":"\\x'),
            b'{"extra":null,' + x[1:], x[:-1] + b',"status":500}', x.replace(b'"status":', b'"Status":'),
            x.replace(b'"bytes":', b'"bytes":-1.5e3,"b2":'), x.replace(b'"host":"', b'"host":"a' + b"b" * 700)])
    return b"\n".join(out) + b"\n"


def take(r):
    import torch
    from warpjq_b200.shard import _DeviceBytes
    return bytes(torch.as_tensor(_DeviceBytes(r.d_out_bytes, max(1, r.out_len)), device="cuda").cpu().numpy()[:r.out_len])


def same(query, got, want):
    if not query.startswith("avg"):
        return got == want
    return abs(float(got) - float(want)) <= 1e-9 * abs(float(want))  # the oracle adds in line order


@pytest.mark.parametrize("rate", RATES)
def test_other_lines_beside_a_template(rate):
    import torch
    import warpjq_b200 as wjq
    data = lines(6_000_000, rate, rate)
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    for query in QUERIES:
        q = wjq.Query(query, chunk_bytes=1 << 20)
        q.set_tiling(1024, 512)
        q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
        r = q.collect_device()
        want = orc.run(query, data)
        assert r.n_lines - r.n_blank == want.stats["lines_in"], query
        assert r.n_invalid == want.stats["malformed"] and r.n_type_error == want.stats["type_errors"], query
        got = q.render_device(r, data) if q.is_aggregate else take(r)
        assert same(query, got, want.out), query
        q.close()


def test_a_template_per_query():
    import torch
    import warpjq_b200 as wjq
    parts = [lines(5_000_000, RATES[i % 3], 40 + i) for i in range(len(QUERIES))]
    offs, total = [], 0
    for p in parts:
        total = (total + 15) & ~15
        offs.append(total)
        total += len(p)
    host = np.zeros(total + 16, dtype=np.uint8)
    for p, o in zip(parts, offs):
        host[o:o + len(p)] = np.frombuffer(p, dtype=np.uint8)
    dev = torch.from_numpy(host).cuda()
    qs = [wjq.Query(x, chunk_bytes=1 << 20) for x in QUERIES]
    for q in qs:
        q.set_tiling(1024, 512)
    for _ in range(2):
        qs[0].batch_launch_mixed(qs, dev.data_ptr(), offs, [len(p) for p in parts],
                                 torch.cuda.current_stream().cuda_stream)
        items, every = qs[0].batch_collect()
        got = wjq.batch_outputs_mixed(qs, items, every, host)
        for query, p, out in zip(QUERIES, parts, got):
            assert same(query, out, orc.run(query, p).out), query
    for q in qs:
        q.close()
