"""Line starts of tiles where a lane classifies more than eight 32-byte chunks:
fewer, as many and more lines a lane than it notes positions for, in one tile
or side by side."""

import random

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


def lines(n_bytes, sizes, seed):
    rng = random.Random(seed)
    out, total = [], 0
    while total < n_bytes:
        pad = max(0, rng.choice(sizes) - 22)
        out.append(b'{"v":%d,"s":"%s"}' % (rng.randrange(1000), b"x" * pad) if pad else rng.choice([b"", b"{}", b"1"]))
        total += len(out[-1]) + 1
    return b"\n".join(out) + rng.choice([b"", b"\n"])


# tile and halo: 8, 9, 18 and 63 chunks a lane
@pytest.mark.parametrize("tiling", [(7168, 512), (8192, 512), (16384, 2048), (61440, 2048)])
@pytest.mark.parametrize("sizes", [[1], [30], [70, 90], [130, 150], [300], [1, 25, 600], [1, 1, 1, 40, 3000]])
def test_line_starts(tiling, sizes):
    import torch
    import warpjq_b200 as wjq
    data = lines(400_000, sizes, sum(sizes) + tiling[0])
    dev = torch.from_numpy(np.frombuffer(data + b"\0" * 16, dtype=np.uint8).copy()).cuda()
    for query in ("sum(.v)", "select(.v < 500) | .v"):
        q = wjq.Query(query, chunk_bytes=1 << 20)
        q.set_tiling(*tiling)
        q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
        r = q.collect_device()
        want = orc.run(query, data)
        assert r.n_lines - r.n_blank == want.stats["lines_in"]
        assert r.n_invalid == want.stats["malformed"] and r.n_type_error == want.stats["type_errors"]
        if q.is_aggregate:
            assert q.render_device(r, data) == want.out
        else:
            from warpjq_b200.shard import _DeviceBytes
            got = bytes(torch.as_tensor(_DeviceBytes(r.d_out_bytes, max(1, r.out_len)), device="cuda").cpu().numpy()[:r.out_len])
            assert got == want.out
        q.close()
