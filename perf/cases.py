"""The work a program has this framework do, as cases that can be timed and compared.

A case names one operation with its sizes and options:

  build   one key set through Context.build: key kind (u64, 16-byte records, pre-hashed
          Keys, strings), keys and results on the device or in numpy arrays
  batch   many key sets in one call (build_batch_flat), device-resident
  serve   a wave of requests through Server.submit / wait, results in host memory
  query   the slots of a key set that was built before (Context.query)
  encode  the compact-vector encoding of a build's result (encode_gpu)

Sizes and parameters are those of the repository's own workloads (sets of 10^3 to 4*2^20
keys, requests of 10^4 to 5*10^7, 10^6 / 10^8 u64 keys, 5*10^7 strings; lambda 5 to 8 with
2048 or 2500 keys per partition), with ragged ones between.  Keys are splitmix64 streams
and printable strings of 8 to 64 bytes, made on the device from the seed.  One context
and one server serve every key set, as in a program that builds many functions: a pass
meets the buffers of another key set than the pass before it.
"""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "phobic-gpu_b200"))
import keygen  # noqa: E402
import phobic  # noqa: E402

KINDS = {"u64": phobic.KEYS_U64, "bytes16": phobic.KEYS_BYTES16, "prehashed": phobic.KEYS_PREHASHED,
         "strings": phobic.KEYS_STRINGS}
KEY_BYTES = {"u64": 8, "bytes16": 16, "prehashed": 16, "strings": 36 + 8}  # strings: mean length + offset
STREAMS = 4                 # of the server
BUDGET = 40 << 30           # device bytes its admitted builds may hold
MAX_REQUEST = 5_000_000     # largest request of a wave


def listed():
    return [
        # The smallest sets of a batch workload, built alone: launches and one partition's chain of tries.
        {"name": "build_u64_1e3", "op": "build", "kind": "u64", "n": 1_000, "lam": 6.0, "P": 2048, "place": "device"},
        # An ordinary small set with a ragged last partition.
        {"name": "build_u64_98765", "op": "build", "kind": "u64", "n": 98_765, "lam": 6.0, "P": 2048,
         "place": "device"},
        # The million-key build of the reference's example size.
        {"name": "build_u64_1e6", "op": "build", "kind": "u64", "n": 1_000_000, "lam": 5.0, "P": 2048,
         "place": "device"},
        # The median request of the served stream, as strings.
        {"name": "build_strings_700001", "op": "build", "kind": "strings", "n": 700_001, "lam": 7.0, "P": 2048,
         "place": "device"},
        # The largest set of a batch workload, 16-byte records (pairs) at the default configuration.
        {"name": "build_pairs_4194301", "op": "build", "kind": "bytes16", "n": 4_194_301, "lam": 8.0, "P": 2048,
         "place": "device"},
        # The headline build.
        {"name": "build_u64_1e8", "op": "build", "kind": "u64", "n": 100_000_000, "lam": 7.0, "P": 2500,
         "place": "device"},
        # The large string build.
        {"name": "build_strings_5e7", "op": "build", "kind": "strings", "n": 50_000_000, "lam": 6.0, "P": 2048,
         "place": "device"},
        # A numpy array of keys into numpy results: the shortest program a user writes.
        {"name": "build_numpy_1e7", "op": "build", "kind": "u64", "n": 10_000_000, "lam": 7.0, "P": 2500,
         "place": "host"},
        # Many sets of very different sizes in one call.
        {"name": "batch_192_sets", "op": "batch", "sets": 192, "lo": 1_000, "hi": 4 << 20, "lam": 6.0, "P": 2048},
        # A burst of requests at the server, 70 % u64 and 30 % strings.
        {"name": "serve_12_requests", "op": "serve", "requests": 12, "lo": 10_000, "hi": MAX_REQUEST, "lam": 7.0,
         "P": 2048},
        # Lookups against a finished function.
        {"name": "query_u64_2e7", "op": "query", "kind": "u64", "n": 20_000_000, "lam": 7.0, "P": 2500},
        # The stored form of the headline build's result.
        {"name": "encode_1e8", "op": "encode", "n": 100_000_000, "lam": 7.0, "P": 2500,
         "pilots": "interleaved_compact", "offsets": "diff"},
    ]


def _log(rng, lo, hi):
    return int(lo * (hi / lo) ** rng.random())


def draw(rng):
    lam, P = rng.choice([5.0, 6.0, 7.0, 8.0]), rng.choice([2048, 2500])
    op = rng.choices(["build", "batch", "serve", "query", "encode"], [12, 2, 1, 2, 1])[0]
    if op == "build":
        kind = rng.choices(["u64", "bytes16", "prehashed", "strings"], [5, 1, 1, 2])[0]
        host = rng.random() < 0.15
        top = 20_000_000 if host else 100_000_000 if kind == "u64" else 50_000_000
        return {"op": op, "kind": kind, "n": _log(rng, 1_000, top), "lam": lam, "P": P,
                "place": "host" if host else "device"}
    if op == "batch":
        sets = _log(rng, 16, 1024)
        return {"op": op, "sets": sets, "lo": _log(rng, 1_000, 10_000), "hi": _log(rng, 50_000, 60_000_000 // sets),
                "lam": lam, "P": P}
    if op == "serve":
        return {"op": op, "requests": rng.randint(4, 16), "lo": _log(rng, 10_000, 100_000),
                "hi": _log(rng, 500_000, MAX_REQUEST), "lam": lam, "P": P}
    if op == "query":
        kind = rng.choices(["u64", "bytes16", "strings"], [3, 1, 1])[0]
        return {"op": op, "kind": kind, "n": _log(rng, 1_000, 50_000_000), "lam": lam, "P": P}
    return {"op": op, "n": _log(rng, 10_000, 100_000_000), "lam": lam, "P": P,
            "pilots": rng.choice(["interleaved_compact", "mono_compact"]), "offsets": rng.choice(["diff", "direct"])}


_handles: dict = {}


def _context():
    if "ctx" not in _handles:
        _handles["ctx"] = phobic.Context(0)
    return _handles["ctx"]


def _server():
    if "srv" not in _handles:
        srv = phobic.Server(0, streams=STREAMS, budget_bytes=BUDGET)
        # Room for a few of the largest requests per stream; results of that many in pageable memory.
        srv.reserve(64 * 4 * MAX_REQUEST, 64 << 20)
        _handles["srv"] = srv
    return _handles["srv"]


def _keys(kind, seed, n):
    """n keys of a kind on the device, from the seed."""
    s = 1_000_003 * (seed + 1)
    if kind == "u64":
        return keygen.splitmix64_cuda(s, n)
    if kind == "strings":
        return keygen.strings_cuda(s, n)
    return keygen.splitmix64_cuda(s, 2 * n).view(n, 2)  # 16 bytes: a pair, or a Key that was hashed before


def _on_host(keys):
    if isinstance(keys, tuple):
        return keys[0].cpu().numpy(), keys[1].cpu().numpy().view(np.uint64)
    return keys.cpu().numpy().view(np.uint64)


def _sizes(case):
    """Sizes of a batch's sets or a wave's requests (the same for every seed: they are the case's)."""
    return keygen.set_sizes(4, case["sets"] if case["op"] == "batch" else case["requests"], case["lo"], case["hi"])


def _result(cfg, n):
    m = cfg.partitions(n)
    return (torch.zeros(cfg.bucketCountPerPartition * m, dtype=torch.int32, device="cuda"),
            torch.zeros(m + 1, dtype=torch.int32, device="cuda"))


def prepare(case, seed):
    cfg = phobic.MPHFconfig(case["lam"], case["P"])
    st = {"case": case, "cfg": cfg, "ctx": _context()}
    op = case["op"]
    if op == "build":
        st["kind"] = KINDS[case["kind"]] if case["kind"] != "strings" else None
        keys = _keys(case["kind"], seed, case["n"])
        st["keys"] = keys if case["place"] == "device" else _on_host(keys)
        st["out"] = _result(cfg, case["n"]) if case["place"] == "device" else None
    elif op == "batch":
        st["sizes"] = _sizes(case)
        st["keys"] = _keys("u64", seed, int(st["sizes"].sum()))
        pstart, ostart = phobic.batch_layout(st["sizes"], cfg)
        st["out"] = (torch.zeros(int(pstart[-1]), dtype=torch.int32, device="cuda"),
                     torch.zeros(int(ostart[-1]), dtype=torch.int32, device="cuda"))
    elif op == "serve":
        st["server"] = _server()
        st["reqs"] = [_keys("strings" if i % 10 in (2, 5, 8) else "u64", 64 * seed + i, int(n))
                      for i, n in enumerate(_sizes(case))]
    else:
        kind = case.get("kind", "u64")
        st["keys"] = _keys(kind, seed, case["n"])
        st["kind"] = KINDS[kind] if kind != "strings" else None
        st["built"] = st["ctx"].build(st["keys"], cfg, out=_result(cfg, case["n"]), kind=st["kind"])
        if op == "encode":
            del st["keys"]
            # Room for every encoding of this many pilots and offsets (at most 4 bytes each, and a header per
            # column): the encoded size depends on the pilots' widths.
            m, B = cfg.partitions(case["n"]), cfg.bucketCountPerPartition
            st["bytes"] = torch.zeros(4 * (B * m + m + 1) + 64 * (B + 2), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    case, cfg, ctx = st["case"], st["cfg"], st["ctx"]
    op = case["op"]
    if op == "build":
        r = ctx.build(st["keys"], cfg, out=st["out"], kind=st["kind"])
        return [r.pilots, r.partition_offsets]
    if op == "batch":
        pilots, offsets, status, _ = phobic.build_batch_flat(ctx, st["keys"], st["sizes"], cfg, *st["out"])
        return [pilots, offsets, status]
    if op == "serve":
        srv = st["server"]
        tickets = [srv.submit(k, cfg) for k in st["reqs"]]
        out = []
        for t in tickets:
            status, r = srv.wait(t)
            out.append([status, r.pilots, r.partition_offsets])
        return out
    if op == "query":
        return ctx.query(st["keys"], cfg, st["built"], kind=st["kind"])
    _, _, size = phobic.encode_gpu(ctx, st["built"], cfg, case["pilots"], case["offsets"], out=st["bytes"])
    return [size, st["bytes"]]


def work(case):
    """Bytes of one pass: keys read once, results written once.  The path computes with
    whole numbers only: it has no floating-point work."""
    cfg = phobic.MPHFconfig(case["lam"], case["P"])
    B = cfg.bucketCountPerPartition

    def built(n):
        m = cfg.partitions(n)
        return 4 * (B * m + m + 1)

    op = case["op"]
    if op == "build":
        b = KEY_BYTES[case["kind"]] * case["n"] + built(case["n"])
    elif op == "batch":
        b = sum(8 * int(n) + built(int(n)) for n in _sizes(case))
    elif op == "serve":
        b = sum(KEY_BYTES["strings" if i % 10 in (2, 5, 8) else "u64"] * int(n) + built(int(n))
                for i, n in enumerate(_sizes(case)))
    elif op == "query":  # keys, the function, one slot per key
        b = (KEY_BYTES[case["kind"]] + 4) * case["n"] + built(case["n"])
    else:  # pilots and offsets in, about 16 bits per pilot out
        b = built(case["n"]) * 3 // 2
    return {"bytes": b, "flops": 0}


def exact(case, seed):
    """Every output is a whole number or a byte, for which equality is the measure."""
    return None
