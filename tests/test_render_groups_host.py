"""Rendering a device result's groups (warpjq_query_render_device, no device):
the output order and text of every key kind, for few groups and for as many
as are sorted and printed by several threads."""

import ctypes
import json
import random

import pytest

import warpjq_b200 as wjq


def keys(n, rng):
    """n distinct (kind, raw text) keys: strings sharing long prefixes, some
    with escapes, numbers spelled differently, literals, arrays."""
    out = [(1, b""), (2, b"true"), (2, b"false"), (3, b"1"), (3, b"1.0"), (3, b"1e0"), (3, b"-0"), (3, b"0"),
           (5, b'["a",1]'), (5, b'["a"]'), (6, b'{"a":1}'), (4, b""), (4, b"a"), (4, b'a,"b'.replace(b'"', b'\\"')),
           (4, b"a\\u0000"), (4, b"caf\\u00e9"), (4, "cafè".encode()), (4, b"abcdefgh"), (4, b"abcdefghi")]
    seen = set(out)
    while len(out) < n:
        k = rng.randrange(4)
        c = ((3, b"%d" % rng.randrange(-10**12, 10**12)) if k == 0 else
             (3, b"%d.%d" % (rng.randrange(1000), rng.randrange(1, 10**9))) if k == 1 else
             (4, b"user-%d" % rng.randrange(10**9)) if k == 2 else
             (4, b"u\\n%d" % rng.randrange(10**9)))
        if c not in seen:
            seen.add(c)
            out.append(c)
    rng.shuffle(out)
    return out[:n]


def order(key):
    kind, raw = key
    if kind == 1:
        return (0, 0.0, b"")
    if kind == 2:
        return (2 if raw == b"true" else 1, 0.0, b"")
    if kind == 3:
        # -0.0 sorts just below 0.0, as the order-preserving bits do
        return (3, (float(raw), 0 if raw.startswith(b"-") else 1), raw)
    if kind == 4:
        return (4, 0.0, json.loads(b'"' + raw + b'"').encode())
    return (5, 0.0, raw)


def text(key):
    kind, raw = key
    if kind == 4:
        s = json.loads(b'"' + raw + b'"')
        return json.dumps(s, ensure_ascii=False).encode()
    return raw if kind != 1 else b"null"


@pytest.mark.parametrize("fmt", ["ndjson", "csv", "count"])
@pytest.mark.parametrize("n", [0, 1, 19, 16383, 16384, 30001])
def test_groups_in_order(n, fmt):
    rng = random.Random(n + 1)
    ks = keys(n, rng)
    q = wjq.Query("group_by(.k) | sum(.v)", fmt, device=False)
    data = bytearray()
    gs = (wjq._GroupExt * max(1, n))()
    for i, (kind, raw) in enumerate(ks):
        gs[i].key_off, gs[i].key_len, gs[i].key_kind = len(data), len(raw), kind
        gs[i].count = gs[i].numeric = i + 1
        gs[i].sum = i * 0.25
        data += raw
    r = wjq.DeviceResult()
    r.groups, r.n_groups = ctypes.cast(gs, ctypes.POINTER(wjq._GroupExt)), n
    got = q.render_device(r, bytes(data) + b"\0" * 16)
    if fmt == "count":
        assert got == b"%d\n" % n
        return
    want = []
    for i in sorted(range(n), key=lambda i: order(ks[i])):
        v = b"%d" % (i // 4) if i % 4 == 0 else repr(i * 0.25).encode()
        if fmt == "ndjson":
            want.append(b'{"k":' + text(ks[i]) + b',"sum":' + v + b"}")
        else:
            cell = json.loads(text(ks[i])).encode() if ks[i][0] == 4 else text(ks[i])
            if any(c in cell for c in b',"\n\r'):
                cell = b'"' + cell.replace(b'"', b'""') + b'"'
            want.append(cell + b"," + v)
    lines = got.split(b"\n")[:-1] if fmt == "ndjson" else None
    if fmt == "csv":
        head, _, got = got.partition(b"\n")
        assert got == b"".join(w + b"\n" for w in want)
    else:
        assert lines == want
