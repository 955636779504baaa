"""The coder's work as its users have it done, for timing.

A case is one call of the public entry points: a whole container compressed or
decompressed (host or device buffers), many buffers in one batched call, the
chunks of a batch coded from a prelearned model, or the fixed-model variant.

Fields of a case:
  op       compress | decompress
  via      host   Context.compress / decompress on host buffers
           dev    Context.compress_dev / decompress_dev on device buffers
           many   Context.compress_many_dev / decompress_many_dev
           model  Context.compress_batch / decompressbatch with a kept Model
           fixed  Context.compress(fixed=True) / decompress, host buffers
  n        input bytes (many: bytes of the largest buffer)
  lo, count  many: smallest buffer and number of buffers, sizes log-uniform
  chunk    bytes per chunk
  unit     bits per unit
  kind     text | walk | random | runs | mixed (64 KiB blocks of the four)

The range is what the command line, the batched calls and the serving loop
meet: buffers from 1 KB to 128 MiB, chunks from 4 KiB to the default 1 MiB,
units of 32 to 256 bits, one chunk to several hundred in flight.
"""
import math

import numpy as np
import torch

import cucm_b200 as cc
from cucm_b200 import workloads as W

KINDS = ("text", "walk", "random", "runs")
BLOCK = 64 << 10
PREFIX = 16 << 10  # bytes the prelearned model is trained on

_kept = {}


def listed():
    return [
        # one small message, one chunk: latency of a single call
        dict(name="compress_4k", op="compress", via="host", n=4096, chunk=4096, unit=128, kind="text"),
        dict(name="decompress_4k", op="decompress", via="host", n=4096, chunk=4096, unit=128, kind="text"),
        # a small file at the default chunk size: the chunk is coded to its
        # full size although the data ends early
        dict(name="compress_small_default", op="compress", via="host", n=20011, chunk=1 << 20, unit=128, kind="text"),
        # a 1 MiB document in 64 KiB chunks: few chunks, most of the chip idle
        dict(name="compress_1m_64k", op="compress", via="host", n=1 << 20, chunk=64 << 10, unit=128, kind="text"),
        dict(name="decompress_1m_64k", op="decompress", via="host", n=1 << 20, chunk=64 << 10, unit=128, kind="text"),
        # a large mixed buffer in 256 chunks, resident in device memory
        dict(name="compress_mixed_128m", op="compress", via="dev", n=128 << 20, chunk=512 << 10, unit=128,
             kind="mixed"),
        dict(name="decompress_mixed_64m", op="decompress", via="dev", n=64 << 20, chunk=256 << 10, unit=128,
             kind="mixed"),
        # a batch of independent buffers of all sizes in one call
        dict(name="compress_many", op="compress", via="many", n=4 << 20, lo=4 << 10, count=48, chunk=64 << 10,
             unit=128, kind="each"),
        dict(name="decompress_many", op="decompress", via="many", n=4 << 20, lo=4 << 10, count=48, chunk=64 << 10,
             unit=128, kind="each"),
        # records coded from a model trained on earlier ones, long units, a
        # ragged last chunk
        dict(name="compress_model_u256", op="compress", via="model", n=777001, chunk=32 << 10, unit=256, kind="text"),
        # the fixed-model variant, each direction
        dict(name="compress_fixed", op="compress", via="fixed", n=16 << 20, chunk=128 << 10, unit=128, kind="text"),
        dict(name="decompress_fixed", op="decompress", via="fixed", n=16 << 20, chunk=128 << 10, unit=128,
             kind="text"),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    via = rng.choice(["host", "host", "dev", "dev", "many", "many", "model", "fixed"])
    op = rng.choice(["compress", "decompress"])
    case = dict(op=op, via=via, kind=rng.choice(["text", "text", "walk", "random", "runs", "mixed", "mixed"]),
                unit=rng.choice([128, 128, 128, 32, 64, 96, 160, 192, 256]))
    chunk = _log(rng, 4 << 10, (512 << 10) if op == "compress" and via != "fixed" else (256 << 10))
    if rng.random() < 0.5:
        chunk = 1 << (chunk.bit_length() - 1)  # as people write them
    case["chunk"] = chunk
    if via == "many":
        case["kind"] = "each"
        case["count"] = rng.randrange(4, 60)
        case["lo"] = _log(rng, 1 << 10, 64 << 10)
        case["n"] = min(_log(rng, 64 << 10, 4 << 20), max(128 << 10, 40 * chunk))
    elif via == "model":
        case["n"] = min(_log(rng, 1000, 1 << 20), 300 * chunk)
    elif via == "fixed":
        case["n"] = max(PREFIX + 1000, min(_log(rng, 64 << 10, 32 << 20), 400 * chunk))
    else:
        case["n"] = min(_log(rng, 1000, 64 << 20), 400 * chunk)
    return case


def _context():
    """The one context that a program keeps for its calls."""
    if "ctx" not in _kept:
        _kept["ctx"] = cc.Context(0)
    return _kept["ctx"]


def _model():
    """The model that a program has trained once on earlier records."""
    if "model" not in _kept:
        _kept["model"] = cc.Model.prelearn(W.text(PREFIX, 7))
    return _kept["model"]


def _bytes(kind, n, seed):
    if kind == "text":
        return W.long_text(n, seed, piece=1 << 20)
    if kind != "mixed":
        return W.make(kind, n, seed)
    rng = np.random.default_rng([seed, 1])
    count = (n + BLOCK - 1) // BLOCK
    kinds = rng.choice(4, size=count, p=[0.5, 0.25, 0.15, 0.10])
    seeds = rng.integers(0, 1 << 62, size=count)
    out = np.empty(n, dtype=np.uint8)

    def fill(i):
        a = i * BLOCK
        k = min(BLOCK, n - a)
        out[a:a + k] = W.make(KINDS[kinds[i]], k, int(seeds[i]))

    W._parallel(fill, range(count))
    return out


def _many_sizes(case):
    """The batch's buffer sizes, the same for every seed: smallest to largest."""
    c = case["count"]
    lo, hi = math.log(case["lo"]), math.log(case["n"])
    return [int(round(math.exp(lo + (hi - lo) * i / (c - 1)))) for i in range(c)]


def _inputs(case, seed):
    if case["via"] != "many":
        return [_bytes(case["kind"], case["n"], seed)]
    rng = np.random.default_rng([seed, 2])
    sizes = _many_sizes(case)
    kinds = rng.choice(4, size=len(sizes), p=[0.5, 0.25, 0.15, 0.10])
    order = np.random.default_rng(len(sizes)).permutation(len(sizes))  # arrival order
    return W._parallel(lambda i: W.make(KINDS[kinds[i]], sizes[order[i]], int(seed) * 1000 + i), range(len(sizes)))


def _cap(case, n):
    if case["via"] == "fixed":  # a model that does not fit its data expands it more
        return 2 * cc.many_cap(n, case["chunk"], PREFIX)
    return cc.many_cap(n, case["chunk"])


def prepare(case, seed):
    ctx = _context()
    data = _inputs(case, seed)
    via, opts = case["via"], dict(chunksize=case["chunk"], unit=case["unit"])
    s = dict(case=case, ctx=ctx, opts=opts)
    if via == "model":
        s["model"] = _model()
        s["in"] = data[0]
        s["out"] = np.zeros(_cap(case, case["n"]), dtype=np.uint8)
        if case["op"] == "decompress":
            s["in"] = ctx.compress_batch(data[0], case["chunk"], case["unit"], s["model"])
        return s
    if via == "fixed":
        opts.update(prelearn=PREFIX, fixed=True)
    if via in ("host", "fixed"):
        s["in"] = data[0]
        s["out"] = np.zeros(_cap(case, data[0].size), dtype=np.uint8)
        if case["op"] == "decompress":
            s["in"] = ctx.compress(data[0], out=s["out"], **opts).copy()
            s["out"] = np.zeros(data[0].size, dtype=np.uint8)
        return s
    s["in"] = [torch.from_numpy(d).cuda() for d in data]
    s["out"] = [torch.zeros(_cap(case, d.size), dtype=torch.uint8, device="cuda") for d in data]
    torch.cuda.synchronize()
    if case["op"] == "decompress":
        packed = run(dict(s, case=dict(case, op="compress")))
        s["in"] = [t[:int(n)].clone() for t, n in zip(packed["out"], packed["n"])]
        s["out"] = [torch.zeros(d.size, dtype=torch.uint8, device="cuda") for d in data]
        torch.cuda.synchronize()
    return s


def run(s):
    """One call.  Containers differ in length from input to input, so the
    caller's whole buffers come back, with the sizes that were written."""
    case, ctx, opts = s["case"], s["ctx"], s["opts"]
    via, pack = case["via"], case["op"] == "compress"
    ins, outs = s["in"], s["out"]
    if via == "model":
        if not pack:
            got = ctx.decompressbatch(ins, case["n"], case["chunk"], case["unit"], s["model"])
            return {"n": len(got), "out": np.frombuffer(got, dtype=np.uint8)}
        got = ctx.compress_batch(ins, case["chunk"], case["unit"], s["model"])
        outs[:len(got)] = np.frombuffer(got, dtype=np.uint8)
        return {"n": len(got), "out": outs}
    if via in ("host", "fixed"):
        got = ctx.compress(ins, out=outs, **opts) if pack else ctx.decompress(ins, out=outs)
        return {"n": got.size, "out": outs}
    ai = [(t.data_ptr(), t.numel()) for t in ins]
    ao = [(t.data_ptr(), t.numel()) for t in outs]
    if via == "dev":
        sizes = [ctx.compress_dev(*ai[0], *ao[0], **opts) if pack else ctx.decompress_dev(*ai[0], *ao[0])]
    else:
        sizes, status = ctx.compress_many_dev(ai, ao, **opts) if pack else ctx.decompress_many_dev(ai, ao)
        if any(status):
            raise RuntimeError("status %s" % status)
    return {"n": np.array(sizes), "out": outs}


def exact(case, seed):
    """Decompression gives the input back; a container has no 64-bit value."""
    if case["op"] == "compress":
        return None
    data = _inputs(case, seed)
    if case["via"] in ("dev", "many"):
        return {"n": np.array([d.size for d in data]), "out": [torch.from_numpy(d) for d in data]}
    return {"n": case["n"], "out": data[0]}


def work(case):
    """Every input byte read (or written) once, the coded bytes the other
    way, and for each of a byte's 8 bits and 8 orders the sector of its slot
    read and, where the model learns, written back; 2 x 8 multiply-adds a bit
    for the prediction and the training."""
    n = sum(_many_sizes(case)) if case["via"] == "many" else case["n"]
    fixed = case["via"] == "fixed"
    return {"bytes": 1.6 * n + n * 64 * (32 if fixed else 64), "flops": n * 8 * 16 * (1 if fixed else 2)}
