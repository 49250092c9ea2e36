"""Groups on the device where a CTA's own record of keys runs out or does not
apply: as many keys as it holds and one more, keys of its longest length and
one byte more, escaped spellings of one key, batches whose inputs share keys,
and values its 32-bit sums do not take (negative, large, fractional, none)."""

import json
import random

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu

QUERIES = ["group_by(.k) | count", "group_by(.k) | sum(.v)", "group_by(.k) | max(.v)", "group_by(.k) | min(.v)",
           "group_by(.k) | avg(.v)"]


def lines(n_keys, key_len, n, seed, values):
    rng = random.Random(seed)
    keys = [("%0*d" % (key_len, i))[-key_len:] if key_len else "" for i in range(n_keys)]
    out = []
    for _ in range(n):
        k = json.dumps(rng.choice(keys))
        if rng.randrange(8) == 0 and len(k) > 2:  # the same key spelled with an escape
            k = '"\\u00%02x' % ord(k[1]) + k[2:]
        out.append('{"k":%s,"v":%s}' % (rng.choice([k] * 12 + ["null", "7", "true"]), rng.choice(values)))
    return ("\n".join(out) + "\n").encode()


VALUES = {"small": ["1", "65535", "65536", "0"], "wide": ["2147483647", "2147483648", "-1", "4294967296"],
          "mixed": ["0.25", "1e3", "null", '"x"', "12", "-0.5"]}


@pytest.mark.parametrize("n_keys", [1, 16, 17, 32, 33, 200])
@pytest.mark.parametrize("key_len", [1, 24, 25])
@pytest.mark.parametrize("values", list(VALUES))
def test_groups_against_the_oracle(n_keys, key_len, values):
    import warpjq_b200 as wjq
    data = lines(min(n_keys, 10 ** key_len), key_len, 6000, n_keys, VALUES[values])
    for q in QUERIES:
        got = wjq.run_bytes(q, data)
        want = orc.run(q, data)
        assert got.rc == want.rc == 0 and got.out == want.out, (q, got.out[:200], want.out[:200])


def test_batch_inputs_share_keys():
    import torch
    import warpjq_b200 as wjq
    inputs = [lines(20, 5, 400, 100 + i, VALUES["small"]) for i in range(24)]
    offs, lens, total = [], [], 0
    for x in inputs:
        total = (total + 15) & ~15
        offs.append(total)
        lens.append(len(x))
        total += len(x)
    host = np.zeros(total, dtype=np.uint8)
    for x, o in zip(inputs, offs):
        host[o:o + len(x)] = np.frombuffer(x, dtype=np.uint8)
    dev = torch.from_numpy(host).cuda()
    for query in QUERIES:
        q = wjq.Query(query, chunk_bytes=1 << 20)
        q.set_tiling(1024, 512)  # several tiles an input, several inputs a CTA
        q.batch_launch(dev.data_ptr(), offs, lens, torch.cuda.current_stream().cuda_stream)
        items, every = q.batch_collect()
        for x, out in zip(inputs, q.batch_outputs(items, every, host)):
            assert out == orc.run(query, x).out, query
        q.close()
