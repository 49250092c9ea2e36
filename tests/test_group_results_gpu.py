"""Group results around the sizes where their way to the host changes: those
that come with the counters, a context's first larger result, later ones in
page-locked room, and more than that room ever holds."""

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


def lines(n):
    """Two lines for each of n keys."""
    return b"".join(b'{"k":%d,"v":%d}\n' % (i % n, i) for i in range(2 * n))


# a context's results one after another: first, second and later ones
@pytest.mark.parametrize("sizes", [[63, 64, 65, 64, 66], [65, 8192, 8193, 20000, 3], [20000, 20001, 65, 1]])
def test_result_sizes(sizes):
    import torch
    import warpjq_b200 as wjq
    query = "group_by(.k) | sum(.v)"
    stream = torch.cuda.current_stream().cuda_stream
    q = wjq.Query(query, chunk_bytes=1 << 20)
    for n in sizes:
        data = lines(n)
        want = orc.run(query, data).out
        dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
        q.launch_device(dev.data_ptr(), len(data), stream)
        r = q.collect_device()
        assert r.n_groups == n and q.render_device(r, data) == want
        assert q.run(data).out == want
        # twice in one batch, the keys of each input its own
        offs, both = [0, (len(data) + 15) & ~15], np.zeros(2 * len(data) + 32, dtype=np.uint8)
        for o in offs:
            both[o:o + len(data)] = np.frombuffer(data, dtype=np.uint8)
        dev = torch.from_numpy(both).cuda()
        q.batch_launch(dev.data_ptr(), offs, [len(data)] * 2, stream)
        items, every = q.batch_collect()
        assert q.batch_outputs(items, every, both) == [want, want]
    q.close()


def test_more_than_page_locked_room():
    import torch
    import warpjq_b200 as wjq
    n = (1 << 20) + 3
    data = lines(n)
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    q = wjq.Query("group_by(.k) | sum(.v)", chunk_bytes=1 << 20)
    for _ in range(2):
        q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
        r = q.collect_device()
        assert r.n_groups == n
        want = b"".join(b'{"k":%d,"sum":%d}\n' % (i, 2 * i + n) for i in range(n))
        assert q.render_device(r, data) == want
    q.close()


def test_collected_again():
    """A run's groups stay where they were handed out until the next launch."""
    import ctypes
    import torch
    import warpjq_b200 as wjq
    data = lines(3000)
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    q = wjq.Query("group_by(.k) | sum(.v)", chunk_bytes=1 << 20)
    for _ in range(3):
        q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
        a, b = q.collect_device(), q.collect_device()
        at = [ctypes.cast(r.groups, ctypes.c_void_p).value for r in (a, b)]
        assert at[0] == at[1] and a.n_groups == b.n_groups == 3000
        assert q.render_device(a, data) == orc.run("group_by(.k) | sum(.v)", data).out
    q.close()
