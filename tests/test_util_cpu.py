"""Runtime services on CPU: logger, trace spans, CRC-32C, watchdogs, deployment config, memory plan."""
import json
import time

import pytest

from dgpp_b200.runtime import rt


def test_logger_levels_and_sink():
    lines = []
    rt.set_log_sink(lines.append)
    rt.set_log_level("warn")
    rt.log("info", "sched", "hidden")
    rt.log("error", "sched", "shown")
    rt.set_log_level("debug")
    rt.log("debug", "kv", "now visible")
    rt.set_log_sink(None)
    rt.set_log_level("info")
    assert len(lines) == 2 and "ERROR [sched] shown" in lines[0] and "DEBUG [kv] now visible" in lines[1]


def test_trace_spans_are_json_lines(tmp_path):
    p = tmp_path / "trace.jsonl"
    assert not rt.trace_enabled()
    rt.trace_open(str(p))
    t0 = rt.trace_now_us()
    rt.trace_emit("prefill", t0, 1234, json.dumps({"tokens": 2048}))
    rt.trace_emit("decode_step", t0 + 2000, 77)
    rt.trace_close()
    rows = [json.loads(l) for l in p.read_text().splitlines()]
    assert [r["name"] for r in rows] == ["prefill", "decode_step"]
    assert rows[0]["dur_us"] == 1234 and rows[0]["args"] == {"tokens": 2048} and rows[1]["args"] == {}


def test_crc32c_known_vectors():
    assert rt.crc32c(b"123456789") == 0xE3069283
    assert rt.crc32c(b"") == 0
    assert rt.crc32c(b"6789", rt.crc32c(b"12345")) == 0xE3069283       # incremental


def test_engine_watchdog_fires_only_on_stall_while_busy():
    fired = []
    w = rt.EngineWatchdog(deadline_ms=150, on_stall=fired.append, poll_ms=20)
    time.sleep(0.3)
    assert not w.fired()                  # idle engine: no deadline
    w.set_busy(True)
    for _ in range(5):
        time.sleep(0.06)
        w.progress()
    assert not w.fired()
    time.sleep(0.4)                       # busy and silent
    assert w.fired() and len(fired) == 1 and fired[0] >= 150
    del w


def test_shutdown_watchdog():
    hit = []
    w = rt.ShutdownWatchdog(limit_ms=100, on_timeout=lambda: hit.append(1))
    time.sleep(0.3)
    assert w.timed_out() and hit == [1]
    w2 = rt.ShutdownWatchdog(limit_ms=200, on_timeout=lambda: hit.append(2))
    w2.disarm()
    time.sleep(0.3)
    assert not w2.timed_out() and hit == [1]


def test_cluster_config_validation_and_digest():
    base = {"model": "acme/tiny", "tensor_parallel": 4, "max_concurrency": 16, "kv_dtype": "fp8"}
    text, d1 = rt.parse_cluster_config(json.dumps(base))
    cfg = json.loads(text)
    assert cfg["tensor_parallel"] == 4 and cfg["prefill_chunk"] == 2048 and cfg["prefix_cache"] is True
    _, d2 = rt.parse_cluster_config(json.dumps({**base, "port": 9000, "host": "0.0.0.0", "log_level": "debug"}))
    assert d1 == d2                                   # per-process settings do not change the digest
    _, d3 = rt.parse_cluster_config(json.dumps({**base, "mtp_depth": 2}))
    assert d3 != d1
    for bad, msg in [({**base, "tensor_paralel": 2}, "unknown key"), ({"port": 1}, "'model' is required"),
                     ({**base, "tensor_parallel": 3}, "tensor_parallel"), ({**base, "kv_dtype": "fp4"}, "kv_dtype"),
                     ({**base, "prefill_chunk": 100}, "prefill_chunk")]:
        with pytest.raises(RuntimeError, match=msg):
            rt.parse_cluster_config(json.dumps(bad))


def test_kv_memory_plan():
    gib = 1 << 30
    blocks, nbytes, tokens = rt.plan_kv(170 * gib, 4 * gib, 8 * gib, 64, 8, 128, 64, True)
    per_block = 64 * 2 * 8 * 64 * (128 + 4)
    assert blocks == (158 * gib) // per_block and nbytes == blocks * per_block and tokens == blocks * 64
    assert rt.plan_kv(2 * gib, 4 * gib, 0, 64, 8, 128, 64) == (0, 0, 0)
    assert rt.plan_kv(170 * gib, 0, 0, 64, 8, 128, 64, True, 1000)[0] == 1000


def test_engine_options_are_config_keys_covered_by_the_digest():
    """Switches that change what the engine computes are `engine_*` keys of the deployment configuration: the
    digest that ranks compare moves with each of them, unknown values are refused, and EngineOptions reads them."""
    from dgpp_b200.engine.options import EngineOptions

    base = {"model": "tiny"}
    text, d0 = rt.parse_cluster_config(json.dumps(base))
    cfg = json.loads(text)
    assert cfg["engine_fp4_splits"] == "auto" and cfg["engine_layer_kernel"] is False
    seen = {d0}
    for k, v in (("engine_decode_splits", 4), ("engine_fuse_combine", False), ("engine_l2_prefetch", True),
                 ("engine_fp4_splits", "resident"), ("engine_cluster_splitk", True), ("engine_fp4_preload", False),
                 ("engine_layer_kernel", True), ("engine_seq_parallel", False), ("engine_moe_prefill_terms", 1),
                 ("engine_mtp_depth", 2), ("engine_pin_split_rows", True)):
        t, d = rt.parse_cluster_config(json.dumps({**base, k: v}))
        assert d not in seen, k
        seen.add(d)
        o = EngineOptions.from_config(json.loads(t))
        assert getattr(o, k[len("engine_"):]) == v
    for bad in ({"engine_fp4_splits": "fast"}, {"engine_decode_splits": -1}, {"engine_unknown": 1}, {"engine_mtp_depth": 4},
                {"engine_moe_prefill_terms": 0}):
        with pytest.raises(Exception):
            rt.parse_cluster_config(json.dumps({**base, **bad}))


def test_process_memory_file_residency_and_prefill_progress(tmp_path):
    from dgpp_b200.runtime import rt

    pm = rt.process_memory()
    assert pm["rss_bytes"] > 1 << 20 and pm["peak_rss_bytes"] >= pm["rss_bytes"] and pm["memlock_limit_bytes"] != 0
    f = tmp_path / "w.bin"
    f.write_bytes(b"x" * (1 << 20))
    frac, size = rt.file_residency(str(f))
    assert size == 1 << 20 and 0.0 <= frac <= 1.0
    assert rt.file_residency(str(tmp_path / "missing"))[0] == -1.0
    p = rt.PrefillProgress()
    p.begin("a", 1000, 0)
    p.begin("b", 50, 10)
    p.advance("a", 256, 40)
    p.advance("a", 100, 90)                 # a smaller count is not an advance
    rows = {r[0]: r for r in p.snapshot(100)}
    assert rows["a"][1:] == (256, 1000, 0, 60) and rows["b"][1:] == (0, 50, 10, 90)
    assert p.most_stalled(100)[0] == "b"
    p.end("b")
    assert p.most_stalled(100)[0] == "a" and len(p.snapshot(100)) == 1


def test_a_kernel_entry_is_typed_before_other_threads_can_find_it(monkeypatch):
    """The table of resolved entries is read without a lock, so an entry must have its argument types when it gets there: ctypes
    passes the pointers of an untyped function as 32-bit integers."""
    from dgpp_b200.ops import _lib

    class Entry:
        def __setattr__(self, key, value):
            assert "dgpp_status_read" not in _lib._FNS, f"visible before its {key} was set"
            object.__setattr__(self, key, value)

    class Lib:
        dgpp_status_read = Entry()

    monkeypatch.setattr(_lib, "_FNS", {})
    monkeypatch.setattr(_lib, "load", Lib)
    fn = _lib._fn("dgpp_status_read")
    assert fn.argtypes == _lib._SIGNATURES["dgpp_status_read"] and fn.restype is _lib.I
    assert _lib._fn("dgpp_status_read") is fn


def test_a_reported_error_sets_the_split_counters_back(monkeypatch):
    """A launch that gave up may leave arrival counts behind; once its error has been raised and cleared the workspaces are at rest."""
    from dgpp_b200.ops import _lib, core as ops

    code = [3]

    def call(name, *args):
        if name == "dgpp_status_read":
            import ctypes as C
            C.cast(args[0], C.POINTER(C.c_int))[0] = code[0]
        elif name == "dgpp_status_clear":
            code[0] = 0

    monkeypatch.setattr(_lib, "call", call)
    ws = ops.GemmWorkspace("cpu", max_partial_floats=16, max_tiles=8)
    ws.counters[2] = 1
    with pytest.raises(RuntimeError, match="code=3"):
        ops.check_status()
    assert not ws.counters.any()
    ws.counters[2] = 1
    ops.check_status()                      # no error: a product may be counting
    assert ws.counters[2] == 1


@pytest.mark.parametrize("rows,shared", [(1, True), (128, True), (129, False), (173, False), (1000, False), (2048, False)])
def test_prompt_products_of_4_bit_weights_share_no_workspace(monkeypatch, rows, shared):
    """Above 128 rows a 4-bit linear neither splits K nor hands the library the device's shared partials and counters, so that callers on
    several streams do not meet there."""
    import torch

    from dgpp_b200.ops import core as ops
    from dgpp_b200.quant.formats import QuantLinear

    seen = []
    monkeypatch.setattr(ops, "_chk", lambda *a: None)
    monkeypatch.setattr(ops, "stream_ptr", lambda *a: 0)
    monkeypatch.setattr(ops, "call", lambda name, *a: seen.append((name, a)))
    ws = ops.GemmWorkspace("cpu", max_partial_floats=16, max_tiles=8)
    monkeypatch.setattr(ops, "default_workspace", lambda dev: ws)
    w = QuantLinear("nvfp4", 5120, 256, torch.zeros(5120, 128, dtype=torch.uint8), scale=torch.zeros(5120, 16, dtype=torch.uint8))
    ops.linear(torch.zeros(rows, 256, dtype=torch.bfloat16), w)
    (name, a), = seen
    assert name == "dgpp_gemm_tc_pair"
    splits, partials, counters = a[13], a[14], a[16]
    assert (splits, partials, counters) == ((0, ws.partials.data_ptr(), ws.counters.data_ptr()) if shared else (1, None, None))


def test_split_counts_of_decode_products():
    """bf16 rows split at most eightfold (what a cluster folds), at every width up to 128 rows alike."""
    from dgpp_b200.ops import core as ops

    for n, k in ((2048, 5632), (1024, 8192), (4096, 4096), (520, 2048)):
        counts = {ops.pick_splits(rows, n, k, ops.pick_bn(rows), most=8) for rows in (1, 16, 17, 33, 64, 128)}
        assert len(counts) == 1 and 1 <= min(counts) <= 8
        assert ops.pick_splits(129, n, k, 256, most=8) == 1
    assert ops.pick_splits(8, 2048, 5632, 16) == 9 and ops.pick_splits(8, 2048, 5632, 16, most=8) == 8


@pytest.mark.parametrize("terms,bn,ctas", [(3, 16, 264), (3, 32, 264), (1, 64, 264), (2, 64, 120), (3, 64, 120)])
def test_cluster_splits_run_in_one_wave(terms, bn, ctas):
    """As many CTAs as an SM's shared memory leaves room for (two of up to 96 columns, one of more), the same count at every row count."""
    from dgpp_b200.ops import core as ops

    for n, k in ((520, 2048), (2048, 5632), (11264, 2048), (5120, 5120), (7168, 5120), (5120, 17408), (34816, 5120)):
        counts = {ops.pick_cluster_splits(rows, n, k, bn, terms) for rows in (1, 8, bn)}
        s, tiles = counts.pop(), -(-n // 128)
        assert not counts and (s == 1 or (s <= 8 and s * tiles <= ctas and k // 256 // s >= 2))


def test_width_of_block_scaled_decode_passes(monkeypatch):
    """Three terms leave the block-scaled kernels above 32 rows; fewer terms, draft rows, the all-reduce push and pinned splits stay."""
    from types import SimpleNamespace

    from dgpp_b200.engine.runner import DenseRunner
    from dgpp_b200.ops import core as ops

    def width(**kw):
        return DenseRunner.fp4_width(SimpleNamespace(**{**dict(fp4_rows=64, act_terms=3, verifies_drafts=False, fuse_ar=False), **kw}))

    assert width() == 32 and width(fp4_rows=8) == 8
    assert width(act_terms=1) == width(act_terms=2) == width(verifies_drafts=True) == width(fuse_ar=True) == 64
    monkeypatch.setattr(ops, "PIN_SPLIT_ROWS", True)
    assert width() == 64
