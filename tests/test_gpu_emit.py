"""The emit pass at the lengths and numbers where its code takes another way (against the CPU restatement), and what it and
the string pool keep from one trace to the next."""
import numpy as np
import pytest

import helpers
from kineto_b200 import synth
from kineto_b200 import tracefile as tf

pytestmark = pytest.mark.gpu


def kernel_records(trace):
    """Copies of a trace's kernel records, and their byte offsets."""
    at, pos = [], 0
    kinds = trace.cupti.view(np.uint32)[::2].tolist()
    while pos < len(kinds):
        if kinds[pos] == tf.KIND_CONCURRENT_KERNEL:
            at.append(pos * 8)
        pos += tf.RECORD_SIZE[kinds[pos]] // 8
    rec = np.stack([trace.cupti[a:a + 208] for a in at]).reshape(-1).view(tf.KERNEL9)
    return rec.copy(), at


def check(trace):
    from kineto_b200 import api
    got, _ = api.process(trace, device=0)
    want, _ = helpers.run_port(trace)
    assert got == want, helpers.first_diff(want, got)


# strings of up to 16 bytes, up to 64, and longer ones each have a way of their own, taken when a whole warp is that short
@pytest.mark.parametrize("low,high", [(1, 1), (15, 16), (17, 17), (7, 64), (64, 65), (65, 72), (95, 97), (1, 130), (300, 5000)])
def test_strings_of_every_kind_at_the_lengths_where_their_way_changes(low, high):
    trace = synth.gen_kernel_launches(700, seed=low * 1000 + high, pool_size=97)
    rng = np.random.default_rng(high)
    pool = trace.pool()
    letters = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz_:<>,0123456789", np.uint8)
    ids = np.array([pool.add(rng.choice(letters, n).tobytes()) for n in [low, high] + rng.integers(low, high + 1, 60).tolist()], np.uint32)
    trace.set_pool(pool)
    kern, at = kernel_records(trace)
    kern["name"] = rng.choice(ids, len(kern))
    cupti = trace.cupti.copy()
    for a, r in zip(at, kern.view(np.uint8).reshape(len(at), 208)):
        cupti[a:a + 208] = r
    trace.cupti = cupti
    trace.op_name = np.where(rng.random(len(trace.op_name)) < 0.5, rng.choice(ids, len(trace.op_name)), trace.op_name).astype(np.uint32)
    md = trace.md.copy()
    string = (md["type"] >= 4) & (rng.random(len(md)) < 0.7)
    md["value"] = np.where(string, rng.choice(ids, len(md)), md["value"])
    md["type"] = np.where(string, rng.choice([4, 5], len(md)), md["type"])
    trace.md = md
    check(trace)


def test_numbers_at_the_edges_of_their_digit_groups():
    trace = synth.gen_kernel_launches(900, seed=61, pool_size=30)
    rng = np.random.default_rng(62)
    kern, at = kernel_records(trace)
    edges = np.array([0, 9, 10, 99, 100, 999, 1000, 1001, 9999, 99999, 100000, 999999, 1000000, 1000001, 999999999, 1000000000,
                      2147483647, 2147483648, 4294967295, 4294967296, 10**12, 10**18, (1 << 64) - 1], np.uint64)
    for name in ("gridX", "gridY", "gridZ", "staticSharedMemory", "registersPerThread", "contextId", "streamId", "graphId", "graphNodeId", "queued",
                 "channelID", "channelType"):
        some = rng.random(len(kern)) < 0.6
        of = edges[:7] if name == "registersPerThread" else edges[:10] if name == "staticSharedMemory" else edges
        kern[name] = np.where(some, rng.choice(of, len(kern)).astype(kern[name].dtype), kern[name])
    kern["end"] = kern["start"] + rng.choice(edges[:14], len(kern))
    cupti = trace.cupti.copy()
    for a, r in zip(at, kern.view(np.uint8).reshape(len(at), 208)):
        cupti[a:a + 208] = r
    trace.cupti = cupti
    check(trace)


# blocks of 64 to 320 threads: a trace that one wave of the chip holds spreads over all SMs
@pytest.mark.parametrize("n", [1, 11, 6_313, 6_315, 31_571, 31_575])
def test_numbers_of_events_at_the_edges_of_the_emit_pass_s_blocks(n):
    check(synth.gen_kernel_launches(n, seed=63, pool_size=20))


def test_pools_in_device_memory_that_grow_and_shrink_between_traces_of_one_context():
    """The context's workspaces are made for a pool as large as the last one; a larger one is done over."""
    import torch
    from kineto_b200 import api
    small = synth.gen_kernel_launches(200, seed=64, pool_size=10)
    large = synth.gen_kernel_launches(200, seed=65, pool_size=3000, name_len=(200, 900))
    ops_only = synth.gen_generic_kernels(300, seed=66, pool_size=2000, name_len=(1000, 3000))  # no CUPTI buffers
    traces = [(t, api.device_arrays(t, "cuda:0"), helpers.run_port(t)[0]) for t in (small, large, ops_only)]
    torch.cuda.synchronize()
    ctx = api.K2J(0)
    for k in (0, 1, 0, 2, 1, 0, 0, 2):
        trace, arrays, want = traces[k]
        ctx.load(trace, arrays)
        ctx.run()
        assert ctx.copy_output().tobytes() == want, k
    ctx.load(small)  # and from host memory behind it
    ctx.run()
    assert ctx.copy_output().tobytes() == traces[0][2]
    ctx.close()


def test_inputs_that_the_default_stream_is_still_writing():
    """Device arrays filled on the legacy default stream just before a load, by a program that does not synchronise: the
    context's first trace and the later ones (which read no sizes back) see them complete."""
    import torch
    from kineto_b200 import api
    trace = synth.gen_kernel_launches(3000, seed=67, pool_size=50)
    want = helpers.run_port(trace)[0]
    full = api.device_arrays(trace, "cuda:0")
    ctx = api.K2J(0)
    for _ in range(3):
        arrays = {k: torch.zeros_like(a) for k, a in full.items()}
        torch.cuda.synchronize()
        assert torch.cuda.current_stream() == torch.cuda.default_stream()
        torch.cuda._sleep(20_000_000)  # some 10 ms
        for k, a in arrays.items():
            a.copy_(full[k])
        ctx.load(trace, arrays)
        ctx.run()
        assert ctx.copy_output().tobytes() == want
    ctx.close()


def test_a_launch_of_no_threads_on_an_unknown_device():
    """Infinite blocks per SM times no threads: not a number, with the sign that x86 gives it."""
    b = synth.TraceBuilder(n_devices=1)
    for i, block in enumerate([(0, 1, 1), (1, 0, 7), (65536, 65536, 1), (32, 1, 1)]):  # (the third product wraps to 0)
        for device in (0, 77):
            b.kernel(b.t0 + 10 * i, b.t0 + 10 * i + 5, 0, "none", device=device, block=block)
    trace = b.build()
    want, _ = helpers.run_port(trace)
    assert want.count(b'"warps per SM": "-nan"') == 3
    check(trace)


def test_slabs_hold_what_the_resident_text_does_for_every_kind_of_kernel_and_copy():
    """Text that leaves slab by slab works out occupancy and rates again: odd launches, an unknown device, copies of any length."""
    import torch
    from kineto_b200 import api
    rng = np.random.default_rng(71)
    trace = synth.gen_mixed(1500, seed=72, pool_size=60, n_devices=4)
    kern, at = kernel_records(trace)
    for name, of in (("registersPerThread", [0, 1, 32, 255, 256, 65535]), ("staticSharedMemory", [0, 1, 48 << 10, 227 << 10, 1 << 30]),
                     ("dynamicSharedMemory", [0, 100, 164 << 10, 1 << 28]), ("blockX", [0, 1, 31, 1024, 4096]), ("gridX", [0, 1, 147, 2**31 - 1]),
                     ("deviceId", [0, 1, 3, 4, 77])):
        kern[name] = np.where(rng.random(len(kern)) < 0.5, rng.choice(np.array(of), len(kern)).astype(kern[name].dtype), kern[name])
    cupti = trace.cupti.copy()
    for a, r in zip(at, kern.view(np.uint8).reshape(len(at), 208)):
        cupti[a:a + 208] = r
    trace.cupti = cupti
    want = helpers.run_port(trace)[0]
    ctx = api.K2J(0)
    text = torch.zeros(len(want) + 1000, dtype=torch.uint8)
    for resident in (False, True, False):
        ctx.load(trace)
        if resident:
            ctx.run()
            got = ctx.copy_output().tobytes()
        else:
            ctx.segment(sync=False)
            got = text[:ctx.emit_to_host(text)["out_bytes"]].numpy().tobytes()
        assert got == want, helpers.first_diff(want, got)
    ctx.close()
