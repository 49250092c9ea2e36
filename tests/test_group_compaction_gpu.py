"""Every group of a run reaches the host: inputs without a malformed line and
with more keys than one warp of the run's last pass compacts, over many tiles,
so that many of its blocks count groups at once."""

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


def lines(n_keys, n, seed):
    """n clean lines over exactly n_keys keys."""
    rng = np.random.default_rng(seed)
    ks = np.concatenate([np.arange(n_keys), rng.integers(0, n_keys, n - n_keys)])
    rng.shuffle(ks)
    return b"".join(b'{"k":"u%d","v":%d}\n' % (k, k % 1000) for k in ks)


@pytest.mark.parametrize("n_keys, n", [(33, 60_000), (3_000, 60_000), (60_000, 200_000), (150_000, 200_000)])
def test_all_groups_are_counted(n_keys, n):
    import torch
    import warpjq_b200 as wjq
    data = lines(n_keys, n, n_keys)
    query = "group_by(.k) | sum(.v)"
    want = orc.run(query, data).out
    assert want.count(b"\n") == n_keys
    assert wjq.run_bytes(query, data).out == want
    stream = torch.cuda.current_stream().cuda_stream
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    q = wjq.Query(query, chunk_bytes=1 << 20)
    q.set_tiling(1024, 512)  # thousands of tiles
    for k in range(40):
        q.launch_device(dev.data_ptr(), len(data), stream)
        r = q.collect_device()
        assert r.n_groups == n_keys, k
    assert q.render_device(r, data) == want
    # the same bytes as the inputs of a batch, cut at line ends
    cuts = [0]
    while cuts[-1] < len(data) and len(cuts) < 5:
        cuts.append(data.index(b"\n", len(data) * len(cuts) // 5) + 1)
    cuts.append(len(data))
    parts = [data[a:b] for a, b in zip(cuts, cuts[1:])]
    offs, total = [], 0
    for p in parts:
        total = (total + 15) & ~15
        offs.append(total)
        total += len(p)
    host = np.zeros(total + 16, dtype=np.uint8)
    for p, o in zip(parts, offs):
        host[o:o + len(p)] = np.frombuffer(p, dtype=np.uint8)
    dev = torch.from_numpy(host).cuda()
    want = [orc.run(query, p).out for p in parts]
    for k in range(10):
        q.batch_launch(dev.data_ptr(), offs, [len(p) for p in parts], stream)
        items, every = q.batch_collect()
        assert [it.n_groups for it in items] == [w.count(b"\n") for w in want], k
    assert q.batch_outputs(items, every, host) == want
    q.close()
