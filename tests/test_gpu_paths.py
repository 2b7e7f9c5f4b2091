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


def _whole_text(ctx, trace):
    """The text of a run, left on the GPU."""
    from kineto_b200 import api
    ctx.load(trace)
    ctx.run()
    ptr, size = ctx.output_ptr()
    return api.device_view(ptr, size, "|u1")


# Sort tiles take one to eight rounds of 256 keys, one more for every 303 104 of them (148 * 8 tiles): the first size of
# three rounds and of eight, the last one of seven, and sizes at and past the last full eight (more tiles than can be
# resident from there on), all but two with a partial last tile.
@pytest.mark.parametrize("n", [606_209, 909_500, 1_400_000, 1_600_001, 2_121_728, 2_121_729, 2_424_832, 2_424_833, 3_000_001])
def test_sort_order_at_every_number_of_rounds(n):
    """Events of one length, so that the sorted text is the unsorted one's rows in numpy's stable order of the starts."""
    import torch
    from kineto_b200 import api
    b = synth.TraceBuilder(n_devices=1, flags=0)
    rec = np.repeat(b.runtime(b.t0, b.t0, 1), n)
    rng = np.random.default_rng(n)
    starts = b.t0 + rng.integers(0, 8_000_000, n) * 1000 + rng.integers(0, 2, n)  # seven digits of microseconds; ties
    rec["start"], rec["end"], rec["correlationId"] = starts, starts + 100, 1_000_000 + np.arange(n)
    trace = b.build()
    trace.cupti, trace.buftab = rec.view(np.uint8), tf.make_buftab(np.arange(n + 1) * rec.itemsize)
    ctx = api.K2J(0)
    rows = _whole_text(ctx, trace)
    length = len(rows) // n
    assert len(rows) == n * length
    rows = rows.view(n, length).clone()
    order = torch.from_numpy(np.argsort(starts, kind="stable")).to("cuda:0")
    got = _whole_text(ctx, cases.with_flags(trace, tf.FLAG_SORT_BY_START))
    assert torch.equal(got.view(n, length), rows[order])
    ctx.close()


# the scan of the event sizes takes two launches up to 4096 * 2048 events, three above; the smallest takes one
@pytest.mark.parametrize("n_events", [200, 4096 * 2048, 4096 * 2048 + 1])
def test_what_the_scan_reports_at_the_edges_of_its_shapes(n_events):
    """Bytes of CPU-op text, the flag of instant events, kernels with collective metadata and the annotations' spans reach
    the host with the scan's totals: a trace whose first op recurs is that op's text as often, then the small trace's."""
    from kineto_b200 import api
    b = synth.TraceBuilder(n_devices=1)
    b.op(b.t0 + 10, b.t0 + 20, 7, "recurs")
    b.op(b.t0 + 10, b.t0 + 900, 8, "record_param_comms", md=[
        ("Collective name", tf.MD_STRING, "allreduce"), ("In msg nelems", tf.MD_INT64, 64), ("Out msg nelems", tf.MD_INT64, 64),
        ("Group size", tf.MD_INT64, 8), ("dtype", tf.MD_STRING, "Float")])
    b.op(b.t0 + 30, b.t0 + 30, 0, "[memory]", type=synth.CPU_INSTANT_EVENT, md=[("Bytes", tf.MD_INT64, 512)])
    b.op(b.t0 + 5, b.t0 + 990, 9, "step", type=synth.USER_ANNOTATION)
    for i in range(40):
        b.extcorr(100 + i, 8)
        b.extcorr(100 + i, 9, ext_kind=tf.EXTERNAL_KIND_CUSTOM1)
        b.runtime(b.t0 + 100 + i, b.t0 + 110 + i, 100 + i)
        b.kernel(b.t0 + 200 + i, b.t0 + 300 + i, 100 + i, "k%d" % i, stream=7 + i % 3)
    small = b.build()
    want = helpers.run_port(small)[0]
    ctx = api.K2J(0)
    assert _whole_text(ctx, small).cpu().numpy().tobytes() == want and ctx.result["annotation_bytes"] > 0
    res0 = dict(ctx.result)
    assert b'"Collective name"' in want[res0["ops_bytes"]:] and b'"ph": "i"' in want
    more = n_events - (small.n_ops + 80)
    for col in ("op_start", "op_end", "op_id", "op_device", "op_resource", "op_thread", "op_type", "op_name", "op_flow", "op_flowt", "op_mdoff"):
        a = getattr(small, col)
        setattr(small, col, np.concatenate([np.repeat(a[:1], more), a]))
    got = _whole_text(ctx, small)
    length = want.index(b"\n  {", 1)
    front = got[:more * length].view(more, length)
    assert bool((front == front[0]).all()) and front[0].cpu().numpy().tobytes() == want[:length]
    assert got[more * length:].cpu().numpy().tobytes() == want
    assert ctx.result["ops_bytes"] == res0["ops_bytes"] + more * length and ctx.result["annotation_bytes"] == res0["annotation_bytes"]
    assert ctx.result["x_events"] == res0["x_events"] + more
    ctx.close()


# the scan of the chunks' class counts (13 columns) takes one launch up to 16 384 chunks of 4 KiB, two above
@pytest.mark.parametrize("n_chunks", [16_384, 16_385])
def test_class_counts_at_the_edge_of_one_launch(n_chunks):
    """A small trace's records over and over: its text as often, and then that of the buffers which make up the number."""
    from kineto_b200 import api
    t = synth.gen_mixed(200, seed=47, pool_size=50, buffer_bytes=4096)
    each, size = t.n_buffers, len(t.cupti)
    times, rest = divmod(n_chunks, each)

    def repeated(k):
        r = tf.Trace(**{attr: getattr(t, attr) for _, attr, _ in tf._SECTIONS})
        tab = np.concatenate([t.buftab.reshape(-1, 2) + np.array([i * size, 0], np.uint64) for i in range(k + 1)])
        r.cupti, r.buftab = np.tile(t.cupti, k + 1), tab[:k * each + rest].reshape(-1)
        return r

    ctx = api.K2J(0)
    alone = repeated(1)
    want = helpers.run_port(alone)[0]
    assert _whole_text(ctx, alone).cpu().numpy().tobytes() == want
    n_ops_text = ctx.result["ops_bytes"]
    first = len(helpers.run_port(t)[0]) - n_ops_text            # text of the records once
    got = _whole_text(ctx, repeated(times))
    body = got[n_ops_text:n_ops_text + times * first].view(times, first)
    assert bool((body == body[0]).all()) and body[0].cpu().numpy().tobytes() == want[n_ops_text:n_ops_text + first]
    assert got[:n_ops_text].cpu().numpy().tobytes() == want[:n_ops_text]
    assert got[n_ops_text + times * first:].cpu().numpy().tobytes() == want[n_ops_text + first:]
    ctx.close()


# one launch serves a column of up to 4096 elements (the tests it calls have the sizes of an earlier limit, of 16 384)
@pytest.mark.parametrize("n", [4095, 4096, 4097])
def test_the_scan_s_one_launch_ends_at_4096_elements(n):
    test_exclusive_scan_at_the_edges_of_its_shapes(n)
    test_class_counts_at_the_edge_of_one_launch(n)
    test_what_the_scan_reports_at_the_edges_of_its_shapes(n)


# of the lanes of a warp that hold one key only the last goes to a join table: keys that recur in a warp, in every warp, hardly ever
@pytest.mark.parametrize("distinct", [1, 2, 31, 700])
def test_join_keys_that_recur(distinct):
    """The last record of a correlation id wins, in each of the two kinds; so does the last op of an id."""
    rng = np.random.default_rng(distinct)
    b = synth.TraceBuilder(n_devices=2, flags=tf.FLAG_USER_ANNOTATIONS)
    for i in range(400):
        b.op(b.t0 + i, b.t0 + 10_000 + i, int(rng.integers(0, distinct + 1)), "op%d" % i,
             type=synth.USER_ANNOTATION if i % 5 == 0 else synth.CPU_OP)
    for i in range(1500):
        b.extcorr(int(rng.integers(0, distinct + 1)), int(rng.integers(0, distinct + 3)),
                  ext_kind=tf.EXTERNAL_KIND_CUSTOM1 if rng.random() < 0.3 else tf.EXTERNAL_KIND_CUSTOM0)
    for i in range(500):
        b.kernel(b.t0 + 20 * i, b.t0 + 20 * i + 15, int(rng.integers(0, distinct + 2)), "k%d" % (i % 7), stream=7 + i % 3)
    trace = b.build()
    from kineto_b200 import api
    got, _ = api.process(trace, device=0)
    want, _ = helpers.run_port(trace)
    assert got == want, helpers.first_diff(want, got)


# lists of up to 4096 spans are ordered by the GPU, longer ones by the host
@pytest.mark.parametrize("n", [4095, 4096, 4097, 6001])
def test_traces_of_many_spans(n):
    """Three annotations over that many spans of (device, stream) rows, first used in any order."""
    from kineto_b200 import api
    rng = np.random.default_rng(n)
    b = synth.TraceBuilder(n_devices=8, flags=tf.FLAG_USER_ANNOTATIONS)
    for a in range(3):
        b.op(b.t0 + a, b.t0 + 1_000_000, 1 + a, "step %d" % a, type=synth.USER_ANNOTATION)
    for i, k in enumerate(np.concatenate([rng.permutation(n), rng.integers(0, n, 500)]).tolist()):
        b.extcorr(1 + i, 1 + k % 3, ext_kind=tf.EXTERNAL_KIND_CUSTOM1)
        b.kernel(b.t0 + 20 * i, b.t0 + 20 * i + 15, 1 + i, "k", device=k // 3 % 8, stream=k // 24)
    trace = b.build()
    want, _ = helpers.run_port(trace)
    assert want.count(b'"cat": "gpu_user_annotation"') == n
    got, _ = api.process(trace, device=0)
    assert got == want, helpers.first_diff(want, got)
