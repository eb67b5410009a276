"""The benchmark's JSON line: every key a reader of it needs, in a few KB."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

X = 1234.567890123456789
PHASES = {k: X for k in ("upload", "parse", "decode", "merge", "drop", "partition", "encode_blocks", "encode_meta",
                         "download")}


def _leg():
    e2e = {"value": X, "unit": "MiB/s", "h2d_bytes_per_step": 1 << 30, "d2h_bytes_per_step": 1 << 30,
           "ms_per_step": X, "jobs_in_flight": 4, "sequential_ms_per_step": X, "sequential_value": X}
    return {"workload": "w" * 150, "input_mib": X, "output_mib": X, "entries_in": 10 ** 7, "entries_out": 10 ** 7,
            "output_files": 16, "steps": 10, "value": X, "unit": "MiB/s", "ms_per_step": X,
            "latency_ms": {"p50": X, "p99": X}, "phase_ms": PHASES, "alg_bytes": PHASES, "per_kernel_gbs": PHASES,
            "e2e": e2e, "pcie": {"h2d_gbs": X, "d2h_gbs": X, "note": "n" * 300},
            "parity": {"checked": True, "files": 16, "against": "a" * 120}, "gpu_launches": 720,
            "roofline": {"bound": "hbm", "kernel": "encode_blocks", "achieved": X, "peak": X, "unit": "GB/s",
                         "frac": 0.5, "traffic": X, "traffic_source": "s" * 80, "per_kernel_frac": PHASES},
            "cpu_baseline": {"value": X, "unit": "MiB/s", "cores": 1, "kind": "port", "sample": "s" * 100}}


def _served(mode):
    slow = [{"latency_ms": X, "queue_ms": X, "phase_ms": PHASES} for _ in range(4)]
    return dict({f"field_{i}": X for i in range(24)}, mode=mode, value=X, unit="MiB/s", p50_ms=X, p99_ms=X,
                slowest=slow, engine={f"stat_{i}": X for i in range(17)})


def _record():
    head = _leg()
    load = {"served": _served("served"), "plain": _served("plain"), "speedup_served_vs_plain": X}
    part = {"value": X, "unit": "MiB/s", "ms_per_step": X, "p50_ms": X, "p99_ms": X, "kernel_launches_per_step": 37.0}
    return dict({k: head[k] for k in ("latency_ms", "parity", "e2e", "pcie", "roofline", "phase_ms", "per_kernel_gbs",
                                      "cpu_baseline", "gpu_launches")},
                metric=bench.METRIC, value=X, unit="MiB/s", n_gpus=1, steps=20, warmup=5, ms_per_step=X,
                higher_is_better=True, scaling="weak", vs_baseline=None, dtype="u8", data="synthetic",
                config={"workload": "w" * 150, "parallelism": "replicas1", "scale": 1.0},
                legs={n: _leg() for n in ("large_B", "l1_l2_at_size", "plain_l0_l1")},
                batched={"workload": "w" * 90, "jobs": 64, "plain": part, "batched": part, "plain_e2e": part,
                         "batched_e2e": part, "speedup_batched_vs_plain": X, "note": "n" * 150},
                served={"workload": "w" * 100, "flushes": 256, "capacity": load, "loads": {"0.5": load, "0.9": load},
                        "note": "n" * 150},
                clocks={"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [], "samples": 3}, host={"cpus": 16})


def test_line_keeps_what_readers_need_in_a_few_kb():
    full = _record()
    line = json.loads(json.dumps(bench.summary_line(full)))
    assert len(json.dumps(full)) > 20000 and len(json.dumps(line)) < 8000
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "clocks", "gpu_launches", "roofline", "parity"):
        want = full[k]
        assert line[k] == want or abs(line[k] - want) < 1e-6 * abs(want) if not isinstance(want, dict) else \
            set(line[k]) == set(want), k
    assert line["served"]["loads"]["0.9"]["plain"]["p99_ms"] == 1234.568
    assert line["legs"]["large_B"]["e2e"]["value"] == 1234.568
    assert line["batched"]["batched"]["value"] == 1234.568


def test_line_without_legs():
    full = dict(_record(), legs={}, batched=None, served=None, pcie=None)
    line = bench.summary_line(full)
    assert line["legs"] == {} and line["batched"] is None and line["served"] is None and line["pcie"] is None
