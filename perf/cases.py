"""The calls of this library whose speed is measured.

Every case is one call as a program that uses the library makes it: a query
over NDJSON (or CSV) held in device memory or in host memory, or over a batch
of device inputs, through the public entry points of `warpjq_b200`, with the
results that such a program takes from it.

A case is a dict:
  via     "device"  launch_device + collect_device (rows stay on the device;
                    group results are rendered to text)
          "host"    Query.run over pageable host memory, output to host memory
          "csv"     CsvConverter.convert on the device, then the device run
          "batch"   batch_launch + batch_collect of one query over many inputs
          "mixed"   batch_launch_mixed: a query per input, from MIXED
  schema  "nginx"   flat access-log lines, fixed key order (the benchmark's)
          "spaced"  the same lines with a blank after each ',' and ':' between
                    members, as json.dumps and most loggers print them
          "nested"  3-5 levels deep, shuffled key order, escapes, 2% malformed
  bytes   the input's size (a batch: its largest input's size)
  query, fmt ("ndjson" or "csv" output), tiled (tiles sized from a sample of
  the input, as the benchmark does, or left at the default), inputs (batches).
"""

import json
import math
import random
import re

import numpy as np
import torch

import warpjq_b200 as wjq

COUNT = "select(.status == 500) | count"
PROJECT = "select(.status >= 500) | {p: .path, b: .bytes}"
BY_HOST = "group_by(.host) | sum(.bytes)"
BY_PATH = "group_by(.path) | max(.latency_ms)"
WHOLE = "select(.status == 500)"
NESTED_PROJECT = 'select(.req.user.tier == "gold" and .resp.code != 200) | {u: .req.user.id, l: .resp.latency}'
NESTED_GROUP = "group_by(.req.user.id) | avg(.resp.latency)"
# The eight queries of a mixed batch, dealt to its inputs.
MIXED = [COUNT, "sum(.bytes)", "max(.latency_ms)", "avg(.latency_ms)", BY_HOST, "group_by(.path) | count",
         PROJECT, WHOLE]
# What else is asked of access logs.
OTHER = ["count", "min(.bytes)", "max(.bytes)", "avg(.latency_ms)", "group_by(.method) | avg(.latency_ms)",
         "group_by(.status) | count", 'select(.method == "POST") | {t: .ts, l: .latency_ms}',
         "select(.bytes > 5000000) | count", "select(.latency_ms > 100) | .path"]

MIB = 1 << 20


def _case(name, via, schema, nbytes, query, fmt="ndjson", tiled=True, inputs=1):
    c = {"via": via, "schema": schema, "bytes": nbytes, "query": query, "fmt": fmt, "tiled": tiled,
         "inputs": inputs}
    return dict(c, name=name) if name else c


def listed():
    return [
        # A handful of fresh log lines polled by a resident service: nothing
        # but launches and latency.
        _case("poll 4 KB", "device", "nginx", 4096, COUNT, tiled=False),
        # One request of a serving mix: rows out, as CSV, at an odd size.
        _case("request 300 KB to csv", "device", "nginx", 300_007, PROJECT, fmt="csv", tiled=False),
        # The plain invocation: 64 MB of a file's bytes in host memory.
        _case("plain 64 MB from host", "host", "nginx", 64_000_000, COUNT),
        # The headline scans over device-resident logs: a counting filter,
        # a selective projection, a low-cardinality aggregate, whole lines.
        _case("count 1 GB", "device", "nginx", 1_000_000_000, COUNT),
        _case("project 768 MB", "device", "nginx", 768_000_001, PROJECT),
        _case("group 1 GB", "device", "nginx", 1_000_000_000, BY_HOST),
        _case("lines 512 MB", "device", "nginx", 512 * MIB, WHOLE),
        # The same kind of log as Python's json module writes it.
        _case("spaced 256 MB", "device", "spaced", 256_000_003, "avg(.latency_ms)"),
        # Structured events of services: nested, shuffled, partly malformed;
        # a filter on nested fields, and a group-by with many keys.
        _case("nested project 256 MB", "device", "nested", 256 * MIB, NESTED_PROJECT),
        _case("nested group 64 MB", "device", "nested", 64 * MIB + 5, NESTED_GROUP),
        # A CSV export queried on the device.
        _case("csv 256 MB", "csv", "nginx", 256 * MIB, BY_PATH),
        # Many small files of uneven size, a query each, in one batch.
        _case("mixed batch of 512", "mixed", "nginx", 2 * MIB, "", inputs=512, tiled=False),
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    """One more case of the same ranges."""
    via = rng.choice(["device"] * 6 + ["host", "csv", "batch", "mixed"])
    flat = MIXED + OTHER
    if via == "device":
        schema = rng.choice(["nginx", "nginx", "spaced", "nested"])
        if schema == "nested":
            q = rng.choice([NESTED_PROJECT, NESTED_GROUP])
            n = _log_uniform(rng, 4096, (64 if q == NESTED_GROUP else 256) * MIB)
        else:
            q = rng.choice(flat)
            n = _log_uniform(rng, 4096, 768 * MIB if schema == "nginx" else 256 * MIB)
        fmt = rng.choice(["ndjson", "ndjson", "csv"])
        if q == WHOLE:
            fmt = "ndjson"  # whole lines have no CSV form
        return _case(None, via, schema, n, q, fmt, rng.random() < 0.7)
    if via == "host":
        return _case(None, via, "nginx", _log_uniform(rng, 4096, 128 * MIB), rng.choice(flat))
    if via == "csv":
        return _case(None, via, "nginx", _log_uniform(rng, 4096, 256 * MIB), rng.choice([BY_PATH, BY_HOST, COUNT, PROJECT, WHOLE]))
    q = rng.choice(["avg(.latency_ms)", COUNT, BY_HOST, WHOLE]) if via == "batch" else ""
    return _case(None, via, "nginx", _log_uniform(rng, 64 << 10, 2 * MIB), q, tiled=False,
                 inputs=_log_uniform(rng, 2, 512))


# -- inputs -----------------------------------------------------------------


def _text(schema, n, seed):
    """About n bytes of whole lines of the schema, as a uint8 array."""
    if schema == "nested":
        buf, used, _ = wjq.gen_nested(n, seed=seed, n_users=1_000_000)
        return buf[:used]
    if schema == "csv":
        buf, used, _ = wjq.gen_nginx_csv(n, seed=seed)
        return buf[:used]
    buf, used, _ = wjq.gen_nginx(n - n // 14 if schema == "spaced" else n, seed=seed)
    if schema == "nginx":
        return buf[:used]
    s = buf[:used].tobytes().replace(b'":', b'": ').replace(b',"', b', "')
    return np.frombuffer(bytearray(s), dtype=np.uint8)


def _spans(case, text, rng):
    """A batch's inputs: consecutive newline-aligned slices of `text` of
    log-uniform size, as (start, end)."""
    spans, pos = [], 0
    for _ in range(case["inputs"]):
        end = pos + _log_uniform(rng, 4096, case["bytes"])
        end += bytes(text[end - 1:end + 4096]).index(b"\n")
        spans.append((pos, end))
        pos = end
    return spans


def _inputs(case, seed):
    """(text, spans, queries) of the case: its bytes on the host, the spans
    of its inputs in them, and the query of each."""
    rng = random.Random(seed)
    if case["via"] in ("batch", "mixed"):
        sizes = random.Random(seed)
        total = sum(_log_uniform(sizes, 4096, case["bytes"]) + 4096 for _ in range(case["inputs"]))
        text = _text("nginx", total + 65536 + total // 256, seed + 1)
        spans = _spans(case, text, rng)
        qs = [case["query"]] * len(spans) if case["via"] == "batch" else \
            [MIXED[rng.randrange(len(MIXED))] for _ in spans]
        return text, spans, qs
    text = _text("csv" if case["via"] == "csv" else case["schema"], case["bytes"], seed + 1)
    return text, [(0, len(text))], [case["query"]]


# An upper bound of the output's share of the input, by query.
_SHARE = {WHOLE: 0.08, PROJECT: 0.03, NESTED_PROJECT: 0.03, NESTED_GROUP: 0.25, OTHER[6]: 0.08, OTHER[8]: 0.02}


def prepare(case, seed):
    text, spans, qs = _inputs(case, seed)
    via = case["via"]
    # the program's own room for the output (its end stays zero)
    size = case["bytes"] * case["inputs"]
    room = int(size * _SHARE.get(case["query"], 0.05 if via == "mixed" else 0.0) * (1.6 if via == "csv" else 1)) + 65536
    st = {"via": via, "host": text, "text": np.zeros(room, dtype=np.uint8)}
    if via == "host":
        st["q"] = wjq.Query(case["query"], case["fmt"])
        return st
    # inputs start on 16-byte boundaries of one device buffer, as the library asks
    offs, lens, total = [], [], 0
    for a, b in spans:
        total = (total + 15) & ~15
        offs.append(total)
        lens.append(b - a)
        total += b - a
    if len(spans) > 1:
        packed = np.zeros(total, dtype=np.uint8)
        for (a, b), o in zip(spans, offs):
            packed[o:o + (b - a)] = text[a:b]
        st["host"] = packed
    dev = torch.empty(total + 16, dtype=torch.uint8, device="cuda")
    dev[:total].copy_(torch.from_numpy(st["host"]))
    st.update(dev=dev, n=total, offs=offs, lens=lens)
    if via == "mixed":
        by_text = {q: wjq.Query(q, chunk_bytes=MIB) for q in MIXED}
        st["qs"] = [by_text[q] for q in qs]
        st["q"] = by_text[MIXED[0]]
        return st
    q = st["q"] = wjq.Query(case["query"], case["fmt"], chunk_bytes=MIB)
    if via == "csv":
        st["conv"] = wjq.CsvConverter()
    elif case["tiled"]:
        q.autotile(st["host"][:MIB])
    if via in ("device", "csv") and not q.is_aggregate:
        st["rows"] = torch.zeros(room, dtype=torch.uint8, device="cuda")
        st["row_off"] = torch.zeros(room // 16, dtype=torch.int64, device="cuda")
        st["line_idx"] = torch.zeros(room // 16, dtype=torch.int64, device="cuda")
    return st


# -- one pass ---------------------------------------------------------------


class _View:
    """Device memory described for torch.as_tensor (no copy)."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _counts(r):
    """The whole numbers of a result (a missing line index as -1)."""
    return np.array([r.n_lines, r.n_blank, r.n_invalid, r.n_type_error, r.n_selected, r.first_invalid,
                     r.first_type_error, r.count, r.numeric, r.isum_lo, r.isum_hi, r.n_int], dtype=np.uint64).view(np.int64)


def _take(to, ptr, n, typestr):
    """Copies n elements of the library's device memory into the program's
    own buffer (the library's is only valid until the next run)."""
    if n:
        to[:n].copy_(torch.as_tensor(_View(ptr, n, typestr), device="cuda"))
    return to


def _text_out(state, text):
    """Text into the program's own buffer."""
    to = state["text"]
    to[:len(text)] = text if isinstance(text, np.ndarray) else np.frombuffer(text, dtype=np.uint8)
    return to


def _result(state, r):
    """A collected result's counts with its values or its rows."""
    q, out = state["q"], {"counts": _counts(r)}
    if q.is_aggregate:
        out["values"] = np.array([r.sum, r.min, r.max])
    else:
        out["rows"] = _take(state["rows"], r.d_out_bytes, r.out_len, "|u1")
        out["row_off"] = _take(state["row_off"], r.d_out_row_off, r.n_selected + 1 if r.n_selected else 0, "<i8")
        out["line_idx"] = _take(state["line_idx"], r.d_out_line_idx, r.n_selected, "<i8")
    return out


def _csv(state, stream):
    conv, q = state["conv"], state["q"]
    conv.reset()
    d, n, _, _ = conv.convert(state["dev"].data_ptr(), state["n"], stream=stream)
    q.launch_device(d, n, stream)
    r = q.collect_device()
    if not q.is_grouped:
        return dict(_result(state, r), length=n)
    # the groups in order of their keys, whose bytes are on the device
    gs = [r.groups[k] for k in range(r.n_groups)]
    ln = [g.key_len for g in gs]
    keys = np.empty(max(1, sum(ln)), dtype=np.uint8)
    conv.gather(d, np.array([g.key_off for g in gs], dtype=np.uint64), np.array(ln, dtype=np.uint32), len(gs), keys,
                stream)
    named = sorted((bytes(keys[e - k:e]), i) for i, (e, k) in enumerate(zip(np.cumsum(ln), ln)))
    values = np.zeros((64, 2))
    values[:len(gs)] = [[gs[i].sum, gs[i].max] for _, i in named]
    return {"counts": _counts(r), "length": n, "group_values": values,
            "text": _text_out(state, b"".join(b"%s,%d\n" % (k, gs[i].count) for k, i in named))}


def run(state):
    q = state["q"]
    if state["via"] == "host":
        r = q.run(state["host"], copy_out=False)
        return {"rc": r.rc, "text": _text_out(state, r.out), "stats": np.array(list(r.stats.values()))}
    stream = torch.cuda.current_stream().cuda_stream
    ptr = state["dev"].data_ptr()
    if state["via"] == "csv":
        return _csv(state, stream)
    if state["via"] == "device":
        q.launch_device(ptr, state["n"], stream)
        r = q.collect_device()
        if q.is_grouped:
            return {"counts": _counts(r), "text": _text_out(state, q.render_device(r, state["host"]))}
        return _result(state, r)
    if state["via"] == "mixed":
        q.batch_launch_mixed(state["qs"], ptr, state["offs"], state["lens"], stream)
        items, every = q.batch_collect()
        texts = wjq.batch_outputs_mixed(state["qs"], items, every, state["host"])
    else:
        q.batch_launch(ptr, state["offs"], state["lens"], stream)
        items, every = q.batch_collect()
        texts = q.batch_outputs(items, every, state["host"])
    return {"counts": np.stack([_counts(it) for it in items]), "lengths": np.array([len(t) for t in texts]),
            "text": _text_out(state, b"".join(texts)), "sums": np.array([it.sum for it in items])}


# -- what it takes, and what it gives in 64 bits ------------------------------


def work(case):
    """Input bytes read once and output bytes written once."""
    if case["via"] in ("batch", "mixed"):
        # the mean of the log-uniform sizes, times the inputs
        hi = case["bytes"]
        n = case["inputs"] * (hi - 4096) / math.log(hi / 4096)
    else:
        n = case["bytes"]
    share = {WHOLE: 0.05, PROJECT: 0.01, NESTED_PROJECT: 0.01}.get(case["query"], 0.0)
    return {"bytes": int(n * (1 + share)), "flops": 0}


_FIELD = {
    "bytes": re.compile(rb'"bytes": ?([0-9]+)'),
    "latency_ms": re.compile(rb'"latency_ms": ?([0-9.]+)'),
}


def _values(query, text):
    """(sum, min, max) of an ungrouped aggregate without a filter over the
    bytes `text`; the ones the aggregate does not give are 0, inf and -inf."""
    m = re.fullmatch(r"(sum|min|max|avg)\(\.(\w+)\)", query)
    if not m:
        return (0.0, math.inf, -math.inf)
    v = [float(x) for x in _FIELD[m.group(2)].findall(text)]
    kind = m.group(1)
    return (math.fsum(v) if kind in ("sum", "avg") else 0.0, min(v) if kind == "min" else math.inf,
            max(v) if kind == "max" else -math.inf)


def exact(case, seed):
    """The floating outputs from plain Python floats (sums rounded once);
    everything else is bytes and whole numbers, which have no rounding."""
    if case["bytes"] > 300 * MIB:
        return None
    text, spans, qs = _inputs(case, seed)
    data = text.tobytes()
    if case["via"] in ("device", "csv") and "group_by" not in case["query"]:
        if case["via"] == "csv" or case["schema"] == "nested" or "|" in case["query"] or case["query"] in (WHOLE, "count"):
            return {"values": np.array(_values("", b""))} if case["query"].endswith("count") else None
        return {"values": np.array(_values(case["query"], data))}
    if case["via"] == "csv" and "group_by" in case["query"]:
        cols = data[:data.index(b"\n")].decode().split(",")
        key = cols.index(re.search(r"group_by\(\.(\w+)\)", case["query"]).group(1))
        kind, field = re.search(r"(sum|max)\(\.(\w+)\)", case["query"]).groups()
        val, by = cols.index(field), {}
        for line in data.split(b"\n")[1:-1]:  # the quoted column is the last
            f = line.split(b",", len(cols) - 1)
            by.setdefault(f[key], []).append(float(f[val]))
        values = np.zeros((64, 2))
        values[:len(by)] = [[math.fsum(by[k]) if kind == "sum" else 0.0, max(by[k]) if kind == "max" else -math.inf]
                            for k in sorted(by)]
        return {"group_values": values}
    if case["via"] in ("batch", "mixed"):
        return {"sums": np.array([_values(q, data[a:b])[0] for q, (a, b) in zip(qs, spans)])}
    return None
