"""What is measured: tANS decode and encode calls through the package's
public entry points, from one 4 KB stream to half a gigabyte.

Symbols are min(255, floor(-ln(U) / lambda)) with U uniform in (0, 1], the
distribution of this repository's benchmark and tests (lambda 0.005 .. 2:
8.6 .. 0.67 bits per symbol), each stream with its own table.  Outputs are
bytes and unit words, equal or wrong: `exact` gives the decoded symbols
straight from the generator.
"""
from __future__ import annotations

import concurrent.futures as cf
import math
import random

import torch

import multians_gb300 as mg
from multians_gb300 import batch, encode, serve

KB, MB = 1 << 10, 1 << 20

# bits per symbol of the table generator's streams over lambda
_BITS = ((0.005, 8.6), (0.05, 6.0), (0.2, 3.83), (1.0, 1.52), (2.0, 0.67))

# the 512 MB stream bounds every drawn size; the walk-heavy statistics
# (long merges: low lambda with a large table) stay at the size listed here
_MAX_PLAIN = 128 * MB


def listed():
    return [
        # the smallest message: a 4 KB record, one blocking drop-in call
        {"name": "decode_4k", "kind": "dropin", "n": 4 * KB + 3, "lam": 0.05, "L": 1024},
        # a page or tile of 128 KB, blocking drop-in call
        {"name": "decode_128k", "kind": "dropin", "n": 128 * KB - 1, "lam": 0.2, "L": 1024},
        # the reference's own demo stream: 16 MB, blocking drop-in call
        {"name": "decode_16m", "kind": "dropin", "n": 16 * MB, "lam": 0.05, "L": 1024},
        # skewed data with a fine table, where decodes synchronise slowest
        {"name": "decode_128m_skewed", "kind": "async", "n": 128 * MB + 77, "lam": 1.0,
         "L": 4096, "source_order": False},
        # the benchmark's headline stream, enqueued on a stream
        {"name": "decode_256m", "kind": "async", "n": 256 * MB, "lam": 0.05, "L": 1024,
         "source_order": False},
        # nearly constant data (0.67 bits per symbol), written in source order
        {"name": "decode_256m_sparse", "kind": "async", "n": 256 * MB - 5, "lam": 2.0,
         "L": 4096, "source_order": True},
        # nearly incompressible data, the largest single stream
        {"name": "decode_512m_dense", "kind": "async", "n": 512 * MB + 1, "lam": 0.005,
         "L": 4096, "source_order": False},
        # many uneven streams with their own tables, planned once and replayed
        {"name": "batch_256", "mix": 11, "kind": "batch", "streams": 256, "lo": 4 * KB, "hi": 4 * MB,
         "lam_lo": 0.01, "lam_hi": 1.0, "wide": False},
        # a handful of small streams of mixed tables in one blocking call
        {"name": "batch_call_48", "mix": 12, "kind": "batch_call", "streams": 48, "lo": KB, "hi": 256 * KB,
         "lam_lo": 0.005, "lam_hi": 2.0, "wide": True},
        # a burst of requests in pinned host memory through the serving loop
        {"name": "serve_64", "mix": 13, "kind": "serve", "streams": 64, "lo": KB, "hi": 8 * MB,
         "lam_lo": 0.005, "lam_hi": 2.0, "wide": True},
        # encoding a small buffer: histogram, table and stream
        {"name": "encode_100k", "kind": "encode", "n": 100_001, "lam": 0.05, "L": 1024},
        # encoding a large buffer with a fine table
        {"name": "encode_64m", "kind": "encode", "n": 64 * MB + 9, "lam": 0.2, "L": 4096},
    ]


def _log_size(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng: random.Random):
    kind = rng.choice(["dropin", "async", "async", "batch", "batch_call", "serve", "encode"])
    L = rng.choice([1024, 2048, 4096])
    lam = round(math.exp(rng.uniform(math.log(0.005), math.log(2.0))), 4)
    if kind == "dropin":
        return {"kind": kind, "n": _log_size(rng, KB, 16 * MB), "lam": lam, "L": L}
    if kind == "async":
        return {"kind": kind, "n": _log_size(rng, 64 * KB, _MAX_PLAIN), "lam": lam, "L": L,
                "source_order": rng.random() < 0.3}
    if kind == "encode":
        return {"kind": kind, "n": _log_size(rng, KB, 64 * MB), "lam": lam, "L": L}
    mix = rng.randrange(1 << 30)
    if kind == "batch":
        return {"kind": kind, "mix": mix, "streams": rng.randint(16, 256), "lo": 4 * KB,
                "hi": _log_size(rng, 256 * KB, 4 * MB), "lam_lo": 0.01, "lam_hi": 1.0,
                "wide": rng.random() < 0.3}
    if kind == "batch_call":
        return {"kind": kind, "mix": mix, "streams": rng.randint(2, 48), "lo": KB,
                "hi": _log_size(rng, 16 * KB, 512 * KB), "lam_lo": 0.005, "lam_hi": 2.0,
                "wide": True}
    return {"kind": kind, "mix": mix, "streams": rng.randint(8, 64), "lo": KB,
            "hi": _log_size(rng, 64 * KB, 8 * MB), "lam_lo": 0.005, "lam_hi": 2.0, "wide": True}


def _symbols(n, lam, seed):
    """n symbols on the GPU, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand(n, generator=g, device="cuda")
    v = (1.0 - u).log_().neg_().div_(lam).floor_().clamp_(max=255.0)
    return v.to(torch.uint8)


def _specs(case, seed):
    """(n, lambda, L, seed) of every stream of a multi-stream case: sizes
    log-uniform and lambda uniform over the case's ranges, the same for every
    seed (the symbols are not)."""
    r = random.Random(case["mix"])
    out = []
    for i in range(case["streams"]):
        n = _log_size(r, case["lo"], case["hi"])
        lam = r.uniform(case["lam_lo"], case["lam_hi"])
        out.append((n, lam, r.choice([1024, 4096]) if case["wide"] else 1024, seed * 4099 + i))
    return out


def _stream(n, lam, L, seed):
    """An encoded stream as a program receives it: units and table on the
    GPU and the scalars of its header."""
    units, n_units, first_bit, first_state, dec = encode.encode(_symbols(n, lam, seed), L)
    return {"units": units.clone(), "n_units": n_units, "n": n, "L": L, "table": dec,
            "d_table": torch.from_numpy(dec.view("int32")).cuda(),
            "first_state": first_state, "first_bit": first_bit}


def _streams(specs):
    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        return list(ex.map(lambda s: _stream(*s), specs))


def _prepare_plain(case, seed):
    s = _stream(case["n"], case["lam"], case["L"], seed)
    s["out"] = torch.empty(s["n"], dtype=torch.uint8, device="cuda")
    if case["kind"] == "dropin":
        s["memory"] = mg.CUHDGPUDecoderMemory(s["n_units"]).allocate()
        return s
    s["cfg"] = {"flags": mg.DECODE_SOURCE_ORDER} if case["source_order"] else {}
    plan = mg.plan(s["n_units"], s["n"], s["L"], s["cfg"])
    s["aux"] = torch.empty(mg.aux_size(s["n_units"], plan), dtype=torch.uint8, device="cuda")
    return s


def _prepare_many(case, seed):
    """Streams with their outputs packed into one buffer."""
    sts = _streams(_specs(case, seed))
    out = torch.empty(sum(s["n"] for s in sts), dtype=torch.uint8, device="cuda")
    descs, at = [], 0
    for s in sts:
        descs.append(batch.desc(s["units"], s["n_units"], out[at: at + s["n"]], s["n"],
                                s["d_table"], s["L"], s["first_state"], s["first_bit"]))
        at += s["n"]
    state = {"streams": sts, "out": out, "descs": descs}
    if case["kind"] == "batch":
        state["batch"] = batch.Batch(descs)
    else:
        state["work"] = torch.empty(batch.Batch.workspace_size(descs), dtype=torch.uint8,
                                    device="cuda")
    return state


def _prepare_serve(case, seed):
    sts = _streams(_specs(case, seed))
    srv = serve.Server(budget_bytes=2 << 30)
    out = torch.empty(sum(s["n"] for s in sts), dtype=torch.uint8).pin_memory()
    reqs, keep, at = [], [], 0
    for i, s in enumerate(sts):
        units = s["units"][: s["n_units"]].cpu().pin_memory()
        keep.append(units)
        reqs.append(serve.request(units, s["n_units"], out[at: at + s["n"]], s["n"],
                                  srv.add_table(s["table"]), s["first_state"], s["first_bit"],
                                  tag=i))
        at += s["n"]
    return {"server": srv, "requests": reqs, "units": keep, "out": out}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("dropin", "async"):
        state = _prepare_plain(case, seed)
    elif kind in ("batch", "batch_call"):
        state = _prepare_many(case, seed)
    elif kind == "serve":
        state = _prepare_serve(case, seed)
    else:
        # the program's own buffer for the stream, as long as it can get
        state = {"symbols": _symbols(case["n"], case["lam"], seed), "L": case["L"],
                 "record": torch.zeros(case["n"] * (case["L"].bit_length() - 1) // 32 + 6,
                                       dtype=torch.int32, device="cuda")}
    state["kind"] = kind
    return state


def run(state):
    kind, s = state["kind"], state
    if kind == "dropin":
        mg.CUHDGPUDecoder.decode(s["units"], s["n_units"], s["out"], s["n"], s["d_table"],
                                 s["memory"], s["first_state"], s["first_bit"], s["L"])
        return s["out"]
    if kind == "async":
        mg.decode_async(s["units"], s["n_units"], s["out"], s["n"], s["d_table"], s["L"],
                        s["first_state"], s["first_bit"], s["aux"], s["cfg"])
        return s["out"]
    if kind == "batch":
        s["batch"].graph_decode(torch.cuda.current_stream())
        return s["out"]
    if kind == "batch_call":
        batch.decode_batch(s["descs"], workspace=s["work"], stream=torch.cuda.current_stream())
        return s["out"]
    if kind == "serve":
        s["server"].submit(s["requests"])
        s["server"].wait(len(s["requests"]))
        return s["out"]
    units, n_units, first_bit, first_state, table = encode.encode(s["symbols"], s["L"])
    s["record"][: n_units + 4].copy_(units)
    return s["record"], n_units, first_bit, first_state, table


def exact(case, seed):
    """Decoded symbols come in decode order, last source symbol first."""
    kind = case["kind"]
    if kind == "encode":
        return None
    if kind in ("dropin", "async"):
        sym = _symbols(case["n"], case["lam"], seed)
        return sym if case.get("source_order") else sym.flip(0)
    out = torch.cat([_symbols(n, lam, sd).flip(0) for n, lam, _, sd in _specs(case, seed)])
    return out.cpu() if kind == "serve" else out


def _stream_bytes(n, lam):
    """Bytes of n symbols encoded and decoded once."""
    x = min(max(math.log(lam), math.log(_BITS[0][0])), math.log(_BITS[-1][0]))
    bits = _BITS[-1][1]
    for (l0, b0), (l1, b1) in zip(_BITS, _BITS[1:]):
        if x <= math.log(l1):
            bits = b0 + (b1 - b0) * (x - math.log(l0)) / (math.log(l1) - math.log(l0))
            break
    return n * (1.0 + bits / 8.0)


def work(case):
    """Each stream read or written once and its symbols likewise; the path
    has no floating-point work."""
    if "n" in case:
        return {"bytes": _stream_bytes(case["n"], case["lam"]) + 4 * case["L"], "flops": 0}
    # sizes log-uniform: the mean is (hi - lo) / ln(hi / lo)
    mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    lam = 0.5 * (case["lam_lo"] + case["lam_hi"])
    return {"bytes": case["streams"] * (_stream_bytes(mean, lam) + 4096), "flops": 0}
