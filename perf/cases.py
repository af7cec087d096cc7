"""What is measured: collectives on CUDA tensors through the public entry points
(`DeviceSession`, `HostAllReduce`), from a three-element metric to the largest
gradient set of the headline benchmark.

One GPU is enough: `ranks` > 1 is a loopback session, in which every rank's part
of a collective runs as grid rows of one launch on this GPU (the same kernels,
host path and barriers as with one GPU per rank; peer memory is local memory).
`ranks` == 1 is the session that a one-GPU job gets from `from_env`.

    listed()            the cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) inputs, session, tensors and views, as a program keeps them
    run(state)          one pass; returns every rank's result
    work(case)          bytes and operations that a pass cannot do without
    tolerance(case)     how far another correct implementation may be off
"""
import math
import random

import torch

from stdml_collective_experimental_b200 import DeviceSession
from stdml_collective_experimental_b200.models.gradsets import gradset_sizes
from stdml_collective_experimental_b200.parallel.host_pipeline import HostAllReduce

DTYPES = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16, "f16": torch.float16,
          "i32": torch.int32, "i64": torch.int64, "u8": torch.uint8}
STAGING = 64 << 20  # what from_env gives a job: two staging slots of 64 MB

# op      all_reduce | group | all_gather | broadcast | host
# memory  heap: tensors in the session's symmetric heap (zero-copy)
#         ordinary: tensors of PyTorch's allocator (staged through the session's slots)
#         registered: the same, reduced where they lie (register_min_bytes = 0)
# count   elements per rank; a group has a gradient set (`set`) instead, or `tensors`
#         ragged tensors of at most `largest` elements each
# scale   "mean": 1 / ranks; "clip": a factor a little below one; "": none


def listed():
    return [
        # loss, correct and seen counts averaged after every step: the smallest call there is
        {"name": "metrics_f32_x8", "op": "all_reduce", "memory": "ordinary", "ranks": 8,
         "dtype": "f32", "count": 3, "reduce": "sum", "scale": "mean", "inplace": True},
        # per-row statistics: integer maximum over an odd count, into another tensor
        {"name": "rowmax_i32_x4", "op": "all_reduce", "memory": "ordinary", "ranks": 4,
         "dtype": "i32", "count": 100_003, "reduce": "max", "scale": "", "inplace": False},
        # one 25 MB gradient bucket of data-parallel training, in the heap
        {"name": "bucket_f32_heap_x8", "op": "all_reduce", "memory": "heap", "ranks": 8,
         "dtype": "f32", "count": 6_553_601, "reduce": "sum", "scale": "mean", "inplace": True},
        # the headline set among 8 ranks: the largest case
        {"name": "bert_base_f32_heap_x8", "op": "group", "memory": "heap", "ranks": 8,
         "dtype": "f32", "set": "bert-base", "wire": "", "scale": "mean"},
        # separately allocated gradients of a convolutional net, no preparation by the user
        {"name": "resnet50_f32_ordinary_x4", "op": "group", "memory": "ordinary", "ranks": 4,
         "dtype": "f32", "set": "resnet50", "wire": "", "scale": "mean"},
        # f32 gradients that travel as bf16
        {"name": "bert_base_wire_bf16_x2", "op": "group", "memory": "ordinary", "ranks": 2,
         "dtype": "f32", "set": "bert-base", "wire": "bf16", "scale": "mean"},
        # bf16 gradients, registered: one launch reduces them where they lie
        {"name": "bert_base_bf16_registered_x8", "op": "group", "memory": "registered", "ranks": 8,
         "dtype": "bf16", "set": "bert-base", "wire": "", "scale": "mean"},
        # shards of activations or of a sharded parameter, a size that no vector divides
        {"name": "shards_f16_gather_x8", "op": "all_gather", "memory": "ordinary", "ranks": 8,
         "dtype": "f16", "count": 1_234_567},
        # a word-embedding table handed to new members
        {"name": "embedding_f32_broadcast_x4", "op": "broadcast", "memory": "ordinary", "ranks": 4,
         "dtype": "f32", "count": 30_522 * 768},
        # the headline benchmark's own call on one GPU
        {"name": "bert_base_f32_heap_x1", "op": "group", "memory": "heap", "ranks": 1,
         "dtype": "f32", "set": "bert-base", "wire": "", "scale": "clip"},
        # the same training script with ordinary gradients, run on one GPU
        {"name": "resnet50_f32_ordinary_x1", "op": "group", "memory": "ordinary", "ranks": 1,
         "dtype": "f32", "set": "resnet50", "wire": "", "scale": "clip"},
        # gradients in pinned host memory: copy in, reduce, copy out
        {"name": "resnet50_f32_host_x1", "op": "host", "memory": "heap", "ranks": 1,
         "dtype": "f32", "count": 25_557_032, "scale": "clip"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _group(rng, **more):
    case = {"op": "group", "scale": "mean", "wire": "", **more}
    if rng.random() < 0.5:
        case["set"] = rng.choice(["resnet50", "resnet50-214", "bert-base", "1024x100", "16384x100", "102400x100"])
    else:
        case.update(tensors=rng.randint(2, 240), largest=_log(rng, 1_000, 4_000_000),
                    set_seed=rng.randrange(1 << 20))
    return case


def draw(rng):
    # a staged or registered set costs more per byte than one in the heap: none that
    # would cost more than the largest listed case
    largest = max(work(c)["bytes"] for c in listed())
    while True:
        case = _draw(rng)
        more = {"ordinary": 3.0, "registered": 1.5}.get(case["memory"], 1.0)
        if work(case)["bytes"] * more <= largest:
            return case


def _draw(rng):
    kind = rng.choice(["small", "bucket", "group_heap", "group_ordinary", "group_wire",
                       "group_registered", "all_gather", "broadcast", "alone", "host"])
    ranks = rng.choice([2, 3, 4, 6, 8])
    if kind == "small":
        return {"op": "all_reduce", "memory": "ordinary", "ranks": ranks,
                "dtype": rng.choice(["f32", "bf16", "f16", "f64", "i32", "i64"]),
                "count": _log(rng, 1, 2_000_000), "reduce": rng.choice(["sum", "sum", "max"]),
                "scale": "", "inplace": False}
    if kind == "bucket":
        return {"op": "all_reduce", "memory": rng.choice(["heap", "ordinary"]), "ranks": ranks,
                "dtype": rng.choice(["f32", "bf16"]), "count": _log(rng, 100_000, 32_000_000),
                "reduce": "sum", "scale": "mean", "inplace": True}
    if kind == "group_heap":
        return _group(rng, memory="heap", ranks=ranks, dtype=rng.choice(["f32", "bf16"]))
    if kind == "group_ordinary":
        return _group(rng, memory="ordinary", ranks=min(ranks, 4), dtype=rng.choice(["f32", "bf16"]))
    if kind == "group_wire":
        return _group(rng, memory="ordinary", ranks=min(ranks, 4), dtype="f32") | {
            "wire": rng.choice(["bf16", "bf16", "f16"])}
    if kind == "group_registered":
        return _group(rng, memory="registered", ranks=ranks, dtype=rng.choice(["f32", "bf16"]))
    if kind == "all_gather":
        return {"op": "all_gather", "memory": rng.choice(["ordinary", "ordinary", "heap"]),
                "ranks": ranks, "dtype": rng.choice(["f32", "bf16", "f16", "u8"]),
                "count": _log(rng, 1, 4_000_000)}
    if kind == "broadcast":
        return {"op": "broadcast", "memory": rng.choice(["ordinary", "ordinary", "heap"]),
                "ranks": ranks, "dtype": rng.choice(["f32", "bf16", "i64"]),
                "count": _log(rng, 1, 24_000_000)}
    if kind == "alone":
        return _group(rng, memory=rng.choice(["heap", "ordinary"]), ranks=1,
                      dtype=rng.choice(["f32", "bf16"])) | {"scale": "clip"}
    return {"op": "host", "memory": "heap", "ranks": 1, "dtype": rng.choice(["f32", "bf16"]),
            "count": _log(rng, 100_000, 26_000_000), "scale": "clip"}


def _sizes(case):
    if "set" in case:
        return gradset_sizes(case["set"])
    rng = random.Random(case["set_seed"])
    return [_log(rng, 1, case["largest"]) for _ in range(case["tensors"])]


def _scale(case):
    return {"mean": 1.0 / case["ranks"], "clip": 0.9995, "": None}[case.get("scale", "")]


def _fill(t, seed):
    """Gradient-sized normal values; small whole numbers for the integer types."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if t.dtype.is_floating_point:
        t.normal_(0.0, 1e-3, generator=g)
    else:
        t.random_(0, 100, generator=g)
    return t


def _session(case, heap_bytes):
    if case["ranks"] == 1:
        return DeviceSession.from_env(rank=0, world=1, device=0, heap_bytes=heap_bytes)
    sess = DeviceSession.loopback(case["ranks"], heap_bytes=heap_bytes, staging_bytes=STAGING)
    if case["memory"] == "registered":
        sess.set_knob("register_min_bytes", 0)
    return sess


def _alloc(sess, case, count, dtype):
    """`count` elements per rank: a list with one tensor for each of the ranks."""
    if case["memory"] == "heap":
        t = sess.symm_empty(count, dtype)
        return t if sess.vranks > 1 else [t]
    return [torch.empty(count, dtype=dtype, device="cuda") for _ in range(case["ranks"])]


def prepare(case, seed):
    dtype = DTYPES[case["dtype"]]
    ranks, op = case["ranks"], case["op"]
    size = torch.empty((), dtype=dtype).element_size()
    state = {"case": case, "scale": _scale(case)}
    if op == "group":
        # tensors start on 16-byte boundaries in the heap (back to back, as a gradient
        # arena lays them out) and on the allocator's 512-byte ones outside it; one flat
        # tensor per rank holds them, so that the result can be handed out as a whole
        sizes = _sizes(case)
        align = (16 if case["memory"] == "heap" else 512) // size
        offsets, total = [], 0
        for n in sizes:
            offsets.append(total)
            total += -(-n // align) * align
    else:
        total = case["count"]
    per_rank = total * (ranks if op == "all_gather" else 1)
    sess = _session(case, (per_rank * size if case["memory"] == "heap" else 0) + (1 << 20))
    state["sess"] = sess
    if op == "host":
        state["in"] = torch.empty(total, dtype=dtype, pin_memory=True)
        state["out"] = torch.empty(total, dtype=dtype, pin_memory=True)
        state["in"].copy_(_fill(torch.empty(total, dtype=dtype, device="cuda"), 64 * seed))
        state["pipe"] = HostAllReduce(sess, total, dtype, chunks=16)
        return state
    if op == "all_gather":
        state["in"] = [torch.empty(total, dtype=dtype, device="cuda") for _ in range(ranks)]
        state["out"] = _alloc(sess, case, per_rank, dtype)
        for t in state["out"]:
            t.zero_()
    else:
        state["in"] = _alloc(sess, case, total, dtype)
    for r, t in enumerate(state["in"]):
        _fill(t, 64 * seed + r)
    if op == "all_reduce" and not case["inplace"]:
        state["out"] = [torch.empty_like(t) for t in state["in"]]
    if op == "group":
        views = [[t[o:o + n] for o, n in zip(offsets, sizes)] for t in state["in"]]
        state["views"] = views if ranks > 1 else views[0]
        state["wire"] = DTYPES[case["wire"]] if case["wire"] else None
    return state


def run(state):
    case, sess = state["case"], state["sess"]
    op = case["op"]
    if op == "group":
        sess.group_all_reduce(state["views"], scale=state["scale"], wire_dtype=state["wire"])
        return state["in"]
    if op == "all_reduce":
        out = state.get("out")
        sess.all_reduce(state["in"], out=out, op=case["reduce"], scale=state["scale"])
        return state["in"] if out is None else out
    if op == "all_gather":
        return sess.all_gather(state["in"], state["out"])
    if op == "broadcast":
        return sess.broadcast(state["in"], root=0)
    return state["pipe"].run(state["in"], state["out"], scale=state["scale"])


def work(case):
    size = torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
    ranks = case["ranks"]
    n = sum(_sizes(case)) if case["op"] == "group" else case["count"]
    if case["op"] == "all_gather":  # every rank's shard read, all of them written on every rank
        return {"bytes": n * size * (ranks + ranks * ranks), "flops": 0}
    if case["op"] == "broadcast":  # the root's tensor read, written on the others
        return {"bytes": n * size * ranks, "flops": 0}
    adds = ranks - 1 + (1 if _scale(case) is not None else 0)
    return {"bytes": 2 * n * size * ranks, "flops": n * adds}


def tolerance(case):
    if case["op"] in ("all_gather", "broadcast") or case.get("reduce") == "max":
        return "exact"
    kind = case.get("wire") or case["dtype"]
    if kind in ("i32", "i64", "u8"):
        return "exact"
    # the order of the additions is free; 16-bit results are rounded once
    return {"rel": {"f64": 1e-14, "f32": 1e-6, "f16": 1e-3, "bf16": 5e-3}[kind]}
