"""Rendering many groups when memory runs out (no device): the call returns
nonzero, from whichever allocation or thread it came, and the process goes on."""

import subprocess
import sys

CHILD = r"""
import ctypes, os, resource
import warpjq_b200 as wjq

n = 60000
q = wjq.Query("group_by(.k) | sum(.v)", device=False)
data = bytearray()
gs = (wjq._GroupExt * n)()
for i in range(n):
    raw = b"%05d-%s\\n" % (i * 7919 % n, b"k" * 60)  # an escape: every key is decoded
    gs[i].key_off, gs[i].key_len, gs[i].key_kind = len(data), len(raw), 4
    gs[i].count = gs[i].numeric = 1
    gs[i].sum = 1.5 * i
    data += raw
r = wjq.DeviceResult()
r.groups, r.n_groups = ctypes.cast(gs, ctypes.POINTER(wjq._GroupExt)), n
data = bytes(data) + b"\0" * 16
h = wjq.libraries()[1]
want = q.render_device(r, data)
out, size = ctypes.c_void_p(), ctypes.c_size_t()
args = (q._q, ctypes.byref(r), ctypes.c_char_p(data), ctypes.byref(out), ctypes.byref(size))
hard = resource.getrlimit(resource.RLIMIT_AS)[1]
refused = 0
for mb in list(range(1, 40)) + [4096]:
    have = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (have + (mb << 20), hard))
    rc = h.warpjq_query_render_device(*args)
    resource.setrlimit(resource.RLIMIT_AS, (hard, hard))
    if rc:
        refused += 1
        assert out.value is None and size.value == 0
    else:
        assert ctypes.string_at(out.value, size.value) == want
        h.warpjq_host_free(out)
assert refused and not rc
print("refused", refused)
"""


def test_out_of_memory_is_an_error():
    p = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, timeout=300)
    assert p.returncode == 0, p.stderr[-600:]
    assert p.stdout.startswith(b"refused")
