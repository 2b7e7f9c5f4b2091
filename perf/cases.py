"""Performance cases: whole traces through the library's public entry points.

A pass is what a program does with one finished trace: it hands the inputs to a context it keeps, runs the pipeline and
takes the text.  Inputs are the seeded synthetic workloads of `kineto_b200.synth`; `via` says how text and inputs travel:

    device   inputs already in HBM, the text stays in HBM (a consumer on the GPU)
    copy     ordinary host arrays in, one host array out: a short on-demand capture
    host     pinned host arrays in, the text leaves slab by slab into one pinned host buffer
    file     ordinary host arrays in, the text is written to a file (in memory: no disk takes part)

A trace is `segments` like intervals of `n` launches (activities, CPU ops ... what the workload's generator counts) one
after the other: the interval is generated, and its ids and times move on from one repetition to the next, as in a capture
of many like iterations.  It ends in some CPU operators that bring its text to a length of the case's own, whatever the seed.
"""
import mmap
import os

import numpy as np
import torch

from kineto_b200 import api, synth
from kineto_b200 import tracefile as tf

DEVICE = "cuda:0"

# Per unit of n, without names pooled once per trace: bytes of the input arrays; bytes of text (means of long traces) and
# how far they stray with the strings that a unit draws.
INPUT_BYTES = {"launches": 373.0, "memory": 447.5, "mixed": 311.8, "op_tree": 661.0, "rank": 395.2, "generic": 85.0}
TEXT_BYTES = {"launches": 1863.0, "memory": 2022.0, "mixed": 1521.0, "op_tree": 3550.0, "rank": 1912.0, "generic": 302.0}
TEXT_STRAYS = {"launches": 115.0, "memory": 115.0, "mixed": 130.0, "op_tree": 260.0, "rank": 115.0, "generic": 52.0}
NAMES = {"launches": 4096, "memory": 4096, "mixed": 8192, "op_tree": 4096, "rank": 4096, "generic": 512}


def _names(case):
    return min(NAMES[case["workload"]], 64 + case["n"] // 4)


def _text_bytes(case):
    """Length of the case's text: the mean of its kind, plus what a seed can add to that, plus the annotations' spans (one
    for each of 8 devices x 32 streams that an annotation meets)."""
    mean, n = TEXT_BYTES[case["workload"]], case["n"]
    strays = 5 * TEXT_STRAYS[case["workload"]] * (_names(case) ** -0.5 + n ** -0.5)
    spans = min(n, 256 * case["annotations"]) * 300 + 500 * case["annotations"]
    return int(case["segments"] * n * (1.004 * mean + strays)) + spans + 8192


def _case(name, workload, n, via="device", segments=1, tsc=False, annotations=0, buffer_kib=4096):
    c = {"workload": workload, "n": n, "via": via, "segments": segments, "tsc": tsc, "annotations": annotations, "buffer_kib": buffer_kib}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest trace anybody looks at: a few operators of a unit test or a micro-benchmark
        _case("launches_150", "launches", 150),
        # one training step, as the profiler delivers it: TSC timestamps, a step annotation, host memory on both ends
        _case("step_2k_copy", "launches", 2_000, "copy", tsc=True, annotations=1),
        # a few steps saved to a trace file
        _case("steps_24k_file", "launches", 24_001, "file", tsc=True, annotations=3),
        # the reference's own benchmark: GPU-kernel activities handed straight to the logger
        _case("generic_100k", "generic", 100_000),
        # a default-length capture with converted timestamps and annotations
        _case("launches_100k_tsc", "launches", 100_003, tsc=True, annotations=10),
        # a million launches, correlation ids shuffled
        _case("launches_1m", "launches", 100_000, segments=10),
        # kernels, copies, memsets and bare runtime calls; odd record counts, buffers that were drained early
        _case("mixed_31k", "mixed", 31_013, buffer_kib=256),
        # the same mix as a long capture: the largest trace here (11.5 M records)
        _case("mixed_3m", "mixed", 150_000, segments=20),
        # the mix from pinned host memory to pinned host memory
        _case("mixed_300k_host", "mixed", 150_000, "host", segments=2),
        # CPU side in front: a tree of nested operators with shape strings and flows
        _case("op_tree_120k", "op_tree", 120_000),
        # an allocator's memory events among the operators
        _case("memory_40k", "memory", 40_009),
        # one rank of a distributed job: collectives with their metadata, events ordered by start time
        _case("rank_250k_sorted", "rank", 125_000, segments=2),
    ]


# Most units of n a drawn trace has, by the way it travels (the listed ones' reach).
_MOST = {"device": {"launches": 1_000_000, "memory": 400_000, "mixed": 3_000_000, "op_tree": 300_000, "rank": 500_000, "generic": 1_000_000},
         "copy": {"launches": 6_000, "memory": 4_000, "mixed": 8_000, "op_tree": 2_500, "rank": 5_000, "generic": 30_000},
         "host": {"launches": 240_000, "memory": 120_000, "mixed": 300_000, "op_tree": 100_000, "rank": 200_000, "generic": 600_000},
         "file": {"launches": 24_000, "memory": 20_000, "mixed": 29_000, "op_tree": 12_000, "rank": 23_000, "generic": 140_000}}


def draw(rng):
    workload = rng.choice(["launches", "launches", "mixed", "mixed", "op_tree", "memory", "rank", "generic"])
    via = rng.choice(["device", "device", "device", "device", "copy", "host", "file"])
    least, most = 100, _MOST[via][workload]
    total = int(round(least * (most / least) ** rng.random()))
    segments = 1 + (total - 1) // 150_000
    tsc = workload == "launches" and segments == 1 and rng.random() < 0.5
    annotations = rng.randint(1, 12) if workload == "launches" and segments == 1 and rng.random() < 0.5 else 0
    return _case("", workload, max(100, total // segments), via, segments, tsc, annotations, rng.choice([64, 256, 1024, 4096, 4096, 4096]))


def _generate(case, seed):
    n, names, kw = case["n"], _names(case), {"buffer_bytes": case["buffer_kib"] << 10}
    if case["workload"] == "launches":
        return synth.gen_kernel_launches(n, seed=seed, pool_size=names, ts_mode=int(case["tsc"]), user_annotations=case["annotations"], **kw)
    if case["workload"] == "memory":
        return synth.gen_kernel_launches(n, seed=seed, pool_size=names, memory_events=0.5, **kw)
    if case["workload"] == "mixed":
        return synth.gen_mixed(n, seed=seed, pool_size=names, **kw)
    if case["workload"] == "op_tree":
        return synth.gen_op_tree(n, seed=seed, pool_size=names, **kw)
    if case["workload"] == "rank":  # sorted by start time: a flag of the trace's parameters
        return synth.gen_distributed_rank(n, seed=seed, pool_size=names, **kw)
    return synth.gen_generic_kernels(n, seed=seed, pool_size=names)


def _record_starts(cupti):
    """{kind: byte offsets of its records}; the generators pack whole records back to back."""
    kinds, at, pos = cupti.view(np.uint32)[::2].tolist(), {}, 0
    slots = {k: size // 8 for k, size in tf.RECORD_SIZE.items()}
    while pos < len(kinds):
        at.setdefault(kinds[pos], []).append(pos)
        pos += slots[kinds[pos]]
    return {k: np.array(v, np.int64) * 8 for k, v in at.items()}


def _repeat(trace, arrays, times):
    """The interval `times` times: correlation ids, op ids, flow ids and times move on, everything else recurs.  `arrays`: the
    interval's arrays on the GPU; they and the trace's buffer table and window become the whole trace's."""
    n_ops, n_md, n_bytes = len(trace.op_start), len(trace.md), trace.cupti.nbytes
    span = int(trace.op_start.max() - trace.op_start.min()) + 1_000_000
    launches = sum(len(v) for k, v in _record_starts(trace.cupti).items() if k == tf.KIND_EXTERNAL_CORRELATION)
    step = torch.arange(times, device=DEVICE).view(-1, 1)
    for k in ("op_start", "op_end", "op_id", "op_device", "op_resource", "op_thread", "op_type", "op_name", "op_flow", "op_flowt"):
        a = arrays[k].view(1, -1).repeat(times, 1)
        if k in ("op_start", "op_end"):
            a += step * span
        elif k == "op_id":
            a += torch.where(a > 0, step * n_ops, 0).to(a.dtype)
        elif k == "op_flow":
            a += torch.where(a > 0, step * int(trace.op_flow.max()), 0).to(a.dtype)
        arrays[k] = a.view(-1)
    arrays["md"] = arrays["md"].repeat(times)
    ends = (arrays["op_mdoff"][1:].view(1, -1) + step * n_md).to(arrays["op_mdoff"].dtype).view(-1)
    arrays["op_mdoff"] = torch.cat([arrays["op_mdoff"][:1], ends])
    cupti = arrays["cupti"].repeat(times)
    if n_bytes:
        wide, narrow = cupti.view(torch.int64).view(times, -1), cupti.view(torch.int32).view(times, -1)
        for kind, at in _record_starts(trace.cupti).items():
            fields = tf.RECORD_DTYPE[kind].fields
            at = torch.from_numpy(at).to(DEVICE)
            for name, by in (("start", span), ("end", span), ("externalId", n_ops)):
                if name in fields:
                    wide[:, (at + fields[name][1]) // 8] += step * by
            narrow[:, (at + fields["correlationId"][1]) // 4] += (step * launches).to(torch.int32)
    arrays["cupti"] = cupti
    tab = np.tile(trace.buftab.reshape(1, -1, 2), (times, 1, 1))
    tab[:, :, 0] += (np.arange(times, dtype=np.uint64) * np.uint64(n_bytes))[:, None]
    trace.buftab = tab.reshape(-1)
    trace.params["window_end_ns"] += (times - 1) * span


# The event of a CPU operator without metadata, as _append_ops makes them, with an empty name.
_OP_TEXT = ('\n  {\n    "ph": "X",\n    "cat": "cpu_op",\n    "name": "",\n    "pid": 424242,\n    "tid": 50000,\n    "ts": 1000000.000,\n'
            '    "dur": 10.000\n    ,\n    "args": {\n      "External id": 1500000000\n    }\n  },')
_OP_NAME = 100


def _append_ops(arrays, first_ns, text_bytes):
    """Appends CPU operators with `text_bytes` of text in all."""
    each = len(_OP_TEXT) + _OP_NAME
    m = text_bytes // each
    if m < 1:
        raise ValueError("the case's text is longer than _text_bytes says")
    last = b"operator".ljust(_OP_NAME + text_bytes - m * each, b".")  # the last one's name takes up what is left
    n_str = len(arrays["pool_off"]) - 1
    pool = torch.from_numpy(np.frombuffer(last[:_OP_NAME] + last, np.uint8).copy()).to(DEVICE)
    ends = int(arrays["pool_off"][-1]) + np.array([_OP_NAME, _OP_NAME + len(last)], np.int64)
    names = np.full(m, n_str)
    names[-1] = n_str + 1
    more = {"pool_data": pool, "pool_off": ends, "op_start": np.full(m, first_ns), "op_end": np.full(m, first_ns + 10_000),
            "op_id": 1_500_000_000 + np.arange(m), "op_device": np.full(m, synth.DEFAULT_PID), "op_resource": np.full(m, 50_000),
            "op_thread": np.full(m, 1_000_000), "op_type": np.full(m, synth.CPU_OP), "op_name": names, "op_flow": np.zeros(m),
            "op_flowt": np.zeros(m), "op_mdoff": np.full(m, int(arrays["op_mdoff"][-1]))}
    for k, a in more.items():
        arrays[k] = torch.cat([arrays[k], torch.as_tensor(a, device=DEVICE).to(arrays[k].dtype)])


def _text_so_far(trace, arrays):
    ctx = api.K2J(0)
    ctx.load(trace, arrays)
    size = ctx.run()["out_bytes"]
    ctx.close()
    return size


def prepare(case, seed):
    trace = _generate(case, seed)
    first_ns = int(trace.op_start.min())
    arrays = api.device_arrays(trace, DEVICE)
    if case["segments"] > 1:
        _repeat(trace, arrays, case["segments"])
    torch.cuda.synchronize()
    _append_ops(arrays, first_ns, _text_bytes(case) - _text_so_far(trace, arrays))
    state = {"via": case["via"], "trace": trace, "ctx": api.K2J(0)}
    if case["via"] == "device":
        torch.cuda.synchronize()
    elif case["via"] == "host":
        arrays = {k: a.cpu().pin_memory() for k, a in arrays.items()}
        state["text"] = torch.empty(_text_bytes(case), dtype=torch.uint8).pin_memory()
    else:
        arrays = {k: a.cpu().numpy() for k, a in arrays.items()}
    state["arrays"] = arrays
    if case["via"] == "file":
        state["file"] = os.fdopen(os.memfd_create("trace.json"), "r+b", buffering=0)
    return state


class _Text:
    """The text in a context's memory; a tensor over it keeps the context alive."""

    def __init__(self, ctx):
        ptr, size = ctx.output_ptr()
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (size,), "typestr": "|u1", "data": (ptr, False), "version": 2}


COUNTS = ("out_bytes", "ops_bytes", "n_records", "x_events", "flow_events", "out_of_range_events", "blocklisted_runtime_events",
          "invalid_external_correlation_events", "unexpected_cuda_events", "in_bytes", "name_bytes", "annotation_bytes")


def run(state):
    ctx, via = state["ctx"], state["via"]
    ctx.load(state["trace"], state["arrays"])
    if via == "host":
        ctx.segment(sync=False)
        result = ctx.emit_to_host(state["text"])
        text = state["text"][:result["out_bytes"]]
    else:
        result = ctx.run()
        if via == "device":
            text = torch.as_tensor(_Text(ctx), device=DEVICE)
        elif via == "copy":
            text = ctx.copy_output()
        else:  # a new file: the one before is cut to nothing
            fd = state["file"].fileno()
            os.ftruncate(fd, 0)
            os.lseek(fd, 0, os.SEEK_SET)
            size = ctx.write_output(fd)
            text = np.frombuffer(mmap.mmap(fd, size, access=mmap.ACCESS_READ), np.uint8)
    return {"text": text, "counts": [result[k] for k in COUNTS]}


def work(case):
    """The input arrays read once, the text written once; a byte of text costs no arithmetic worth counting."""
    return {"bytes": case["n"] * case["segments"] * INPUT_BYTES[case["workload"]] + _text_bytes(case), "flops": 0}


def tolerance(case):
    return "exact"  # text and counts
