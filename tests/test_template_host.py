"""Line templates (warpjq_b200/csrc/walker.cuh build_template and
walk_template), compiled for the host, against the oracle: a line that a
template decides gets the oracle's verdict and values, whichever valid line
the template was made from, and the lines of one shape are decided by it."""

import ctypes
import os
import random
import subprocess

import pytest

from oracle import pyoracle as orc
from tests import corpus

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "native", "template_host.cc")
OUT = os.path.join(HERE, "native", "_build", "libtemplate_host.so")


@pytest.fixture(scope="module")
def harness():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    deps = [SRC, os.path.join(HERE, "native", "walker_host.cc")] + \
        [os.path.join(ROOT, "warpjq_b200", "csrc", f) for f in ("walker.cuh", "devutil.cuh", "plan.h", "plan_build.h")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-o", OUT, SRC,
                        os.path.join(ROOT, "warpjq_b200", "csrc", "host", "query.cc")], check=True)
    L = ctypes.CDLL(OUT)
    L.th_eval.argtypes = [ctypes.c_char_p, ctypes.c_char_p, ctypes.c_size_t, ctypes.c_size_t,
                          ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_size_t),
                          ctypes.POINTER(ctypes.c_size_t), ctypes.POINTER(ctypes.c_int)]
    L.wh_free.argtypes = [ctypes.c_void_p]
    o = orc.lib()
    o.oracle_eval_lines.argtypes = [ctypes.c_char_p, ctypes.c_char_p, ctypes.c_size_t,
                                    ctypes.POINTER(ctypes.c_void_p), ctypes.POINTER(ctypes.c_size_t)]
    return L, o


def check(harness, data, query, start):
    """(lines, lines the template decided, whether there was one)."""
    L, o = harness
    p, n = ctypes.c_void_p(), ctypes.c_size_t()
    assert o.oracle_eval_lines(query.encode(), data, len(data), ctypes.byref(p), ctypes.byref(n)) == 0
    want = ctypes.string_at(p.value, n.value).split(b"\n")
    o.oracle_free(p)
    hits, made = ctypes.c_size_t(), ctypes.c_int()
    assert L.th_eval(query.encode(), data, len(data), start, ctypes.byref(p), ctypes.byref(n), ctypes.byref(hits),
                     ctypes.byref(made)) == 0
    got = ctypes.string_at(p.value, n.value).split(b"\n")
    L.wh_free(p)
    for i, (a, b) in enumerate(zip(got, want)):
        assert a == b, f"`{query}` line {i} (template from {start}):\n template: {a[:300]!r}\n oracle: {b[:300]!r}"
    assert len(got) == len(want)
    return len(want) - 1, hits.value, made.value


def edited(lines, rng, count):
    """Lines with random byte edits around and inside their values."""
    out = []
    for _ in range(count):
        b = bytearray(rng.choice(lines))
        for _ in range(rng.randrange(1, 3)):
            at = rng.randrange(len(b))
            k = rng.randrange(3)
            if k == 0:
                b[at:at] = bytes([rng.choice(b'"\\{}[]:,0123456789.eE+-tu \t\r\x01\xc3')])
            elif k == 1:
                del b[at]
            else:
                b[at] = rng.choice(b'"\\{}[]:, \x01ua0')
        out.append(bytes(b).replace(b"\n", b" "))
    return out


FLAT = ["select(.status == 500) | count", "select(.status >= 500) | {p: .path, b: .bytes}",
        "group_by(.host) | sum(.bytes)", ".ua", "count", "select(.latency_ms > 50) | .method", ".", ".status.x"]


@pytest.mark.parametrize("query", FLAT)
@pytest.mark.parametrize("spaced", [False, True])
def test_lines_of_one_shape(harness, query, spaced):
    import warpjq_b200 as wjq
    buf, used, _ = wjq.gen_nginx(150_000, seed=8)
    data = bytes(buf[:used])
    if spaced:
        data = data.replace(b'":', b'": ').replace(b',"', b', "')
    lines = data.split(b"\n")[:-1]
    extra = edited(lines, random.Random(3), 800)
    all_, hits, made = check(harness, data, query, 5)
    # a path through a scalar is missing or a type error, by the value: no template
    assert made == (query != ".status.x") and hits == (all_ if made else 0)
    check(harness, b"\n".join(lines[:50] + extra) + b"\n", query, 7)


@pytest.mark.parametrize("start", range(0, 60, 3))
def test_template_of_any_line(harness, golden, start):
    """Templates of hostile and nested lines, tried on every other line."""
    import warpjq_b200 as wjq
    sb, su, _ = wjq.gen_nested(30_000, seed=4, n_users=100)
    nested = bytes(sb[:su])
    for q in ['select(.req.user.tier == "gold" and .resp.code != 200) | {u: .req.user.id, l: .resp.latency}',
              ".meta.trace.span.id", ".req.user", ".resp.code[0]"]:
        check(harness, nested + b"\n".join(edited(nested.split(b"\n")[:-1], random.Random(start), 200)) + b"\n", q, start)
    hostile = corpus.corpus(11, 200, 0.1)
    for q in golden["diff_queries"][start % 5::5]:
        check(harness, hostile, q, start)


def test_limits(harness):
    """Shapes at and past a template's limits: values, literal sizes, depth,
    duplicate keys, arrays, objects as values, lone scalars."""
    def line(keys, v=b"1"):
        return b"{" + b",".join(b'"%s":%s' % (k, v) for k in keys) + b"}"
    many = [b"k%d" % i for i in range(40)]
    shapes = [line(many[:23]), line(many[:24]), line([b"a" * n for n in (1, 120, 121, 122)]), line([b"a" * 200]),
              line([b"a", b"a"]), b'{"a":' * 8 + b"1" + b"}" * 8, b'{"a":' * 9 + b"1" + b"}" * 9, b'{"a":[1]}',
              b'{"a":{}}', b'{"a":{"b":1}}', b"{}", b"5", b'"a"', b"[]", b'{"a":"x"}', b'{"a":""}', b'{"a":null}',
              b'{ "a" :\t1 , "b" : "x\\u00e9\\n" } ', b'{"a":1}\r', b'{"\\u0061":1}', line(many[:11], b'"x"')]
    data = b"\n".join(s for s in shapes for _ in range(2)) + b"\n"
    for q in [".a", ".a.b", "count", ".k1", "select(.a == 1)", "group_by(.a) | count", ".a[0]"]:
        for k in range(len(shapes)):
            check(harness, data, q, 2 * k)
