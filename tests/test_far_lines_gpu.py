"""Lines longer than their window: the search for their newline, from every
offset within a 16-byte block, to a newline in every place of one, and to the
input's end."""

import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("end", [b"\n", b"", b"\r\n"])
@pytest.mark.parametrize("lead", [0, 1, 7, 15])
def test_far_line_ends(lead, end):
    import torch
    import warpjq_b200 as wjq
    import numpy as np
    # windows of 1,536 bytes; the long lines end 0 .. 40 bytes past one
    body = [b'{"p":"%s"}' % (b"p" * lead)]
    for k in range(41):
        body.append(b'{"v":%d,"s":"%s"}' % (k, b"y" * (1500 + k)))
        body.append(b'{"v":%d,"s":"%s' % (k, b"z" * (1560 + k)))  # cut: malformed
        body.append(b'{"v":1}')
    body.append(b'{"v":5,"s":"%s"}' % (b"w" * 5000))
    data = b"\n".join(body) + end
    dev = torch.from_numpy(np.frombuffer(data + b"\n" * 16, dtype=np.uint8).copy()).cuda()
    q = wjq.Query("sum(.v)", chunk_bytes=1 << 20)
    q.set_tiling(1024, 512)
    q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
    r = q.collect_device()
    want = orc.run("sum(.v)", data)
    assert q.render_device(r, data) == want.out
    assert r.n_invalid == want.stats["malformed"] == 41 and r.n_lines - r.n_blank == want.stats["lines_in"]
    q.close()
