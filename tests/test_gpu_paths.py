"""Paths that are chosen by size or by record class, at the sizes where the choice changes (results against numpy or the
CPU restatement)."""
import numpy as np
import pytest

import cases
import helpers
from kineto_b200 import synth
from kineto_b200 import tracefile as tf

pytestmark = pytest.mark.gpu


# one launch up to 2 tiles of 8192; two launches up to 4096 tiles of 2048; three above
@pytest.mark.parametrize("n", [1, 8192, 16384, 16385, 2048 * 9 + 1, 4096 * 2048, 4096 * 2048 + 1])
def test_exclusive_scan_at_the_edges_of_its_shapes(n):
    import torch
    from kineto_b200 import api
    sizes = np.random.default_rng(n).integers(0, 1 << 20, n, dtype=np.uint32)
    d_sizes = torch.from_numpy(sizes.view(np.int32)).to("cuda:0")
    d_off = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda:0")
    torch.cuda.synchronize()
    ctx = api.K2J(0)
    total = ctx.exclusive_scan(d_sizes, d_off[:n])
    ctx.close()
    sums = np.cumsum(sizes, dtype=np.uint64)
    off = d_off.cpu().numpy()
    assert total == int(sums[-1]) and off[0] == 0 and off[n] == -1
    assert np.array_equal(off[1:n].astype(np.uint64), sums[:-1])


def test_device_rows_that_change_between_calls_of_one_context():
    """Equal device rows are not uploaded again; changed ones are, and so is the way back."""
    from kineto_b200 import api
    a = synth.gen_kernel_launches(300, seed=41, pool_size=20)
    b = synth.gen_kernel_launches(300, seed=41, pool_size=20)
    b.devprops = b.devprops.copy()
    b.devprops["num_sms"] = 7
    b.devprops["max_threads_per_sm"] = 1024
    want = {id(t): helpers.run_port(t)[0] for t in (a, b)}
    assert want[id(a)] != want[id(b)]
    ctx = api.K2J(0)
    for t in (a, a, b, b, a):
        ctx.load(t)
        ctx.run()
        assert ctx.copy_output().tobytes() == want[id(t)]
    ctx.close()


# a tile of the sort is one round of 256 keys up to 148 * 8 of them (303 104 keys, two a launch), two rounds above
@pytest.mark.parametrize("n", [151_552, 151_553])
def test_sorted_trace_at_the_edge_of_the_sort_s_tiles(n):
    from kineto_b200 import api
    trace = cases.with_flags(synth.gen_kernel_launches(n, seed=43, pool_size=50), tf.FLAG_SORT_BY_START)
    got, res = api.process(trace, device=0)
    want, _ = helpers.run_port(trace)
    assert got == want, helpers.first_diff(want, got)


# up to 4096 spans are ordered in pinned memory that earlier runs have filled, more of them in a list of their own
@pytest.mark.parametrize("n", [3, 4095, 4096, 5000])
def test_appended_spans_that_name_an_annotation_twice(n):
    """Parts of two shards handed over without merging: of the entries of one (device, stream, op) the one used first is
    written, once, and nothing that an earlier run left behind."""
    from kineto_b200 import api
    trace = cases.annotation_trace()
    once = np.zeros(n - 1, api.SPAN)
    once["start_ns"] = int(trace.params["window_start_ns"][0]) + 10 * np.arange(n - 1)
    once["end_ns"] = once["start_ns"] + 7
    once["first_event"] = np.arange(n - 1)
    once["device"], once["stream"], once["op_id"] = 1, np.arange(n - 1) // 2, np.arange(n - 1) % 2
    again = once[:1].copy()
    again["first_event"], again["start_ns"] = n, again["start_ns"] + 3
    texts = []
    for spans in (once, np.concatenate([once, again]), np.concatenate([again, once])):
        ctx = api.K2J(0)
        ctx.load(trace)
        before = ctx.run()["out_bytes"]
        assert ctx.result["annotation_bytes"] > 0
        added = ctx.append_spans(spans)
        text = ctx.copy_output().tobytes()
        ctx.close()
        assert len(text) == before + added
        texts.append(text[before:])
    assert texts[0].count(b'"ph": "X"') == n - 1
    assert texts[1] == texts[0] and texts[2] == texts[0]


def test_a_shard_without_events_has_no_parts_of_spans():
    """The parts of an earlier run of the same context are not reported for a shard that holds nothing to write."""
    import torch
    from kineto_b200 import api
    full = cases.annotation_trace()
    b = synth.TraceBuilder(n_devices=2, flags=tf.FLAG_USER_ANNOTATIONS)
    b.extcorr(1, 20, ext_kind=tf.EXTERNAL_KIND_CUSTOM1)   # a record that no event comes from
    ctx = api.K2J(0)
    for trace in (full, b.build()):
        ctx.load(trace)
        info = ctx.segment()
        ext = api.device_view(info.external_records, int(info.n_external) * 2, "<i8").clone()
        ops = torch.from_numpy(trace.op_id.astype(np.int32)).to("cuda:0")
        torch.cuda.synchronize()
        ctx.set_global_join(ext, int(info.n_external), 0, ops, trace.n_ops)
        out = ctx.emit()["out_bytes"]
        parts = ctx.partial_spans()
        assert (len(parts) > 0) == (out > 0) == (trace is full)
    ctx.close()
