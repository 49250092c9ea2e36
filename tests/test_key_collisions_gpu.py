"""Keys whose 32-bit hashes are the same but whose bytes are not, short enough
for a CTA's own record and longer, in an input that ends with its last key's
line: they are told apart wherever keys are compared."""

import numpy as np
import pytest

from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


def hashes(keys):
    """The group table's hash of equally long byte strings (an array of their
    bytes), up to the last step, which maps no two values to one."""
    n, size = keys.shape
    padded = np.zeros((n, -(-size // 4) * 4), dtype=np.uint8)
    padded[:, :size] = keys
    h = np.full(n, 0x811C9DC5, dtype=np.uint32)
    for w in padded.view("<u4").T:
        h = (h ^ w) * np.uint32(0x9E3779B1)
        h ^= h >> np.uint32(15)
    return h


def colliding(size, seed):
    """Keys of `size` bytes of which every one shares its hash with another."""
    rng = np.random.default_rng(seed)
    keys = np.full((1 << 18, size), ord("k"), dtype=np.uint8)
    keys[:, -12:] = rng.integers(ord("a"), ord("z") + 1, (len(keys), 12), dtype=np.uint8)
    keys = np.unique(keys, axis=0)
    h = hashes(keys)
    order = np.argsort(h, kind="stable")
    twin = np.zeros(len(keys), dtype=bool)
    eq = h[order][1:] == h[order][:-1]
    twin[order[1:][eq]] = twin[order[:-1][eq]] = True
    return [bytes(k) for k in keys[twin]]


@pytest.mark.parametrize("size", [12, 23, 24, 25, 31, 40])
def test_colliding_keys(size):
    import torch
    import warpjq_b200 as wjq
    keys = colliding(size, size)
    assert len(keys) >= 2
    rng = np.random.default_rng(size)
    body = [b'{"k":"%s","v":%d}' % (keys[i], v) for i, v in zip(rng.integers(0, len(keys), 4000), rng.integers(0, 9, 4000))]
    for lead in range(4):  # the keys at every offset within a word, the last one's line without a newline
        data = b'{"k":"%s"}\n' % (b"x" * lead) + b"\n".join(body)
        dev = torch.from_numpy(np.frombuffer(data, dtype=np.uint8).copy()).cuda()
        for query in ("group_by(.k) | count", "group_by(.k) | sum(.v)"):
            q = wjq.Query(query, chunk_bytes=1 << 20)
            q.set_tiling(1024, 512)
            q.launch_device(dev.data_ptr(), len(data), torch.cuda.current_stream().cuda_stream)
            r = q.collect_device()
            assert q.render_device(r, data) == orc.run(query, data).out, (size, lead, query)
            q.close()
