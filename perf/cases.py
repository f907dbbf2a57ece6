"""The codec's performance cases: what a program that uses this library has
it do, through its public calls, from single small buffers to the largest
ones and batches of many.

A case is a dict of plain values:

  op         "compress" / "decompress": compress_into / decompress_into, one
             device buffer per call on a kept workspace;
             "frame": frame_compress then frame_decompress, which size their
             results and check the device status on the host;
             "ans_encode" / "ans_decode": the byte coder's drop-in calls;
             "batch_compress" / "batch_decompress": many buffers in one call.
  data       the values (generators of mans_b200.workloads, or a kind of raw
             bytes): each stands for a kind of array the codec is used on.
  n          elements (single-buffer ops).
  p          probability bits of the coder (9, 10 or 11).
  layout     mapped-buffer layout of uint16 (0 native, 1 V12, 2 CPU-V2).
  count, hi  batch ops: number of buffers and the largest buffer's bytes;
             sizes are log-uniform between 4 KiB and hi, uint16 and uint32
             buffers alternating.
"""
from __future__ import annotations

import math

import torch

import mans_b200 as mb
from mans_b200 import workloads as W
from mans_b200.batch import Batch

# Stream bytes per input byte of each kind of data (they are a property of
# the data and the format, the same for every implementation of it).
RATIO = {"laplace_u16": 0.555, "gradient_u16": 0.684, "volume_u16": 0.645, "quant_u32": 0.430,
         "detector_u32": 0.334, "skewed": 0.753, "uniform": 1.03, "two": 0.086, "sparse": 0.396}
ELEM = {"laplace_u16": 2, "gradient_u16": 2, "volume_u16": 2, "quant_u32": 4, "detector_u32": 4,
        "skewed": 1, "uniform": 1, "two": 1, "sparse": 1}
DTYPE = {1: torch.uint8, 2: torch.uint16, 4: torch.uint32}
LAPLACE_MAX = 8 << 20  # bytes; drawn on the host


def listed():
    return [
        # The smallest request of a stream of detector tiles (16 KiB): launches and
        # latency are all of it.
        {"name": "small_u16_compress", "op": "compress", "data": "gradient_u16", "n": 8192, "p": 10,
         "layout": 0},
        # A ragged buffer of quantisation codes stored as a self-describing frame and
        # put in an archive buffer and read back, sizes returned to the host.
        {"name": "frame_u32_roundtrip", "op": "frame", "data": "quant_u32", "n": 250_001, "p": 10,
         "layout": 0},
        # One tomography-like buffer of 4,194,304 values (8 MiB), both directions.
        {"name": "tomo_u16_compress", "op": "compress", "data": "laplace_u16", "n": W.C1_N, "p": 10,
         "layout": 0},
        {"name": "tomo_u16_decompress", "op": "decompress", "data": "laplace_u16", "n": W.C1_N,
         "p": 10, "layout": 0},
        # A run of 16 detector frames of 4096 x 4096 uint32 (1 GiB), both directions.
        {"name": "detector_u32_compress", "op": "compress", "data": "detector_u32", "n": W.C2_N,
         "p": 10, "layout": 0},
        {"name": "detector_u32_decompress", "op": "decompress", "data": "detector_u32", "n": W.C2_N,
         "p": 10, "layout": 0},
        # A 2048 x 2048 x 256 uint16 volume (2 GiB), the largest single buffer.
        {"name": "volume_u16_compress", "op": "compress", "data": "volume_u16", "n": W.C4_N, "p": 10,
         "layout": 0},
        {"name": "volume_u16_decompress", "op": "decompress", "data": "volume_u16", "n": W.C4_N,
         "p": 10, "layout": 0},
        # Raw bytes (already mapped elsewhere, or text-like) through the byte coder
        # alone at its highest precision, an odd size.
        {"name": "bytes_ans_encode", "op": "ans_encode", "data": "skewed", "n": 100_000_007, "p": 11},
        {"name": "bytes_ans_decode", "op": "ans_decode", "data": "skewed", "n": 100_000_007, "p": 11},
        # What a server folds into one launch: buffers of 4 KiB to 64 MiB of both
        # element types, about 1.6 GB, both directions.
        {"name": "batch_mixed_compress", "op": "batch_compress", "count": 256, "hi": 64 << 20, "p": 10},
        {"name": "batch_mixed_decompress", "op": "batch_decompress", "count": 256, "hi": 64 << 20,
         "p": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["compress", "decompress", "compress", "decompress", "frame", "ans_encode",
                     "ans_decode", "batch_compress", "batch_decompress"])
    p = rng.choice([9, 10, 10, 10, 11])
    if op.startswith("batch"):
        return {"op": op, "count": _log_int(rng, 4, 256), "hi": _log_int(rng, 256 << 10, 64 << 20),
                "p": p}
    if op.startswith("ans"):
        return {"op": op, "data": rng.choice(["skewed", "skewed", "sparse", "two", "uniform"]),
                "n": _log_int(rng, 4 << 10, 256 << 20), "p": p}
    data = rng.choice(["laplace_u16", "gradient_u16", "volume_u16", "quant_u32", "detector_u32"])
    lo, hi = 16 << 10, 1 << 30
    if data == "laplace_u16":
        hi = LAPLACE_MAX
    if op == "frame":
        hi = 16 << 20 if data != "laplace_u16" else LAPLACE_MAX
    layout = rng.choice([0, 0, 0, 1, 2]) if ELEM[data] == 2 else 0
    return {"op": op, "data": data, "n": _log_int(rng, lo // ELEM[data], hi // ELEM[data]), "p": p,
            "layout": layout}


# ---------------------------------------------------------------- inputs
def _values(data, n, seed):
    """n values of the given kind on the GPU."""
    if ELEM[data] == 1:
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        if data == "uniform":
            return torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)
        u = torch.rand(n, device="cuda", generator=g)
        if data == "two":
            return torch.where(u < 0.9, 3, 250).to(torch.uint8)
        q = 0.05 if data == "skewed" else 0.3  # geometric, from 0
        k = torch.log1p(-u).div_(math.log1p(-q)).floor_()
        return k.clamp_(0, 255).to(torch.uint8)
    m = -(-n // 2048) * 2048 if data == "volume_u16" else n
    x = W.gen_device(data, m, seed)
    return x if m == n else x[:n].clone()


def _capacity(nbytes):
    """Room for a stream: a program that keeps what does not compress as it is
    gives the codec little more than the input's bytes."""
    return nbytes + nbytes // 8 + (64 << 10)


def _compress(case, x, ws):
    out = torch.zeros(_capacity(x.numel() * x.element_size()), dtype=torch.uint8, device="cuda")
    size = torch.zeros(1, dtype=torch.int64, device="cuda")
    mb.compress_into(ws, x, out, size, case["p"], layout=case["layout"])
    ws.check()
    return out, size


def _batch_plan(case):
    """Buffers of the case: element bytes, elements and offset in one pool."""
    items, off = [], 0
    for i, s in enumerate(W.mixed_sizes(case["count"], 3, 4 << 10, case["hi"]).tolist()):
        elem = 2 if i % 2 == 0 else 4
        n = s // elem - 37 * i % 509  # uneven tails
        items.append({"elem": elem, "n": n, "bytes": n * elem, "off": off,
                      "a": 800.0 - 13.0 * (i % 100), "b": 17.0 * (i % 90) - 700.0})
        off += -(-s // 256) * 256
    return items, off


def _batch_inputs(case, seed):
    plan, total = _batch_plan(case)
    pool = W.gen_mixed_device(plan, total, seed)
    xs = [pool[i["off"]:i["off"] + i["bytes"]].view(DTYPE[i["elem"]]) for i in plan]
    caps = [-(-_capacity(i["bytes"]) // 256) * 256 for i in plan]
    out = torch.zeros(sum(caps), dtype=torch.uint8, device="cuda")
    outs = list(torch.split(out, caps))
    sizes = torch.zeros(len(xs), dtype=torch.int64, device="cuda")
    return xs, out, outs, sizes, total


def prepare(case, seed):
    op = case["op"]
    if op.startswith("batch"):
        xs, out, outs, sizes, total = _batch_inputs(case, seed)
        b = Batch(case["count"], total)
        items = Batch.compress_items(xs, outs, sizes, case["p"])
        if op == "batch_compress":
            return {"op": op, "batch": b, "items": items, "keep": xs, "out": out, "sizes": sizes}
        b.compress_async(items)
        b.check(len(xs))
        shapes = [(x.numel(), x.dtype) for x in xs]
        lens = [-(-n * d.itemsize // 256) * 256 for n, d in shapes]
        back = torch.zeros(sum(lens), dtype=torch.uint8, device="cuda")
        backs = [t[:n * d.itemsize].view(d) for t, (n, d) in zip(torch.split(back, lens), shapes)]
        streams = [o[:n].clone() for o, n in zip(outs, sizes.tolist())]
        return {"op": op, "batch": b,
                "items": Batch.decompress_items(streams, [s.numel() for s in streams], backs),
                "keep": streams, "bytes": back}
    x = _values(case["data"], case["n"], seed)
    nbytes = x.numel() * x.element_size()
    if op.startswith("ans"):
        out = torch.zeros(mb.getMaxCompressedSize(nbytes), dtype=torch.uint8, device="cuda")
        size = torch.zeros(1, dtype=torch.int32, device="cuda")
        state = {"op": op, "p": case["p"], "x": x, "out": out, "size": size}
        if op == "ans_decode":
            mb.ansEncode(case["p"], x, x.numel(), out, size)
            state = {"op": op, "p": case["p"], "stream": out[:int(size.item())].clone(),
                     "back": torch.zeros_like(x)}
            state["bytes"] = state["back"]
        return state
    ws = mb.Workspace(max(nbytes, 1))
    state = {"op": op, "p": case["p"], "layout": case["layout"], "ws": ws}
    if op == "decompress":
        out, size = _compress(case, x, ws)
        stream = out[:int(size.item())].clone()
        del out
        del x
        back = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
        return {**state, "stream": stream, "back": back.view(DTYPE[ELEM[case["data"]]]), "bytes": back}
    state["x"] = x
    if op == "frame":
        state["archive"] = torch.zeros(_capacity(nbytes), dtype=torch.uint8, device="cuda")
    if op == "compress":
        state["out"] = torch.zeros(_capacity(nbytes), dtype=torch.uint8, device="cuda")
        state["size"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    op = state["op"]
    if op == "compress":
        mb.compress_into(state["ws"], state["x"], state["out"], state["size"], state["p"],
                         layout=state["layout"])
        return state["out"], state["size"]
    if op == "decompress":
        mb.decompress_into(state["ws"], state["stream"], state["stream"].numel(), state["back"],
                           layout=state["layout"])
        return state["bytes"]
    if op == "frame":
        frame = mb.frame_compress(state["x"], state["p"], state["layout"], state["ws"])
        state["archive"][:frame.numel()].copy_(frame)
        return (state["archive"], frame.numel(),
                mb.frame_decompress(frame, state["ws"]).view(torch.uint8))
    if op == "ans_encode":
        mb.ansEncode(state["p"], state["x"], state["x"].numel(), state["out"], state["size"])
        return state["out"], state["size"]
    if op == "ans_decode":
        mb.ansDecode(state["p"], state["stream"], state["back"])
        return state["bytes"]
    if op == "batch_compress":
        state["batch"].compress_async(state["items"])
        return state["out"], state["sizes"]
    state["batch"].decompress_async(state["items"])
    return state["bytes"]


def work(case):
    """Bytes a pass reads and writes once each: values and stream."""
    if case["op"].startswith("batch"):
        plan, _ = _batch_plan(case)
        total = sum(i["bytes"] * (1 + RATIO["gradient_u16" if i["elem"] == 2 else "quant_u32"])
                    for i in plan)
        return {"bytes": float(total), "flops": 0.0}
    once = case["n"] * ELEM[case["data"]] * (1 + RATIO[case["data"]])
    return {"bytes": float(once * (2 if case["op"] == "frame" else 1)), "flops": 0.0}
