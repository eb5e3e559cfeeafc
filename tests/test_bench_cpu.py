"""Host logic of the benchmark's measurement loop (no GPU): the visiting order the reference uses
(qual/src/device_benchmark.rs:1228-1239) and how many graph launches make one sample."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("bench_under_test", os.path.join(ROOT, "bench.py"))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def test_measurement_order_rotates_and_reverses():
    order = _bench().Protocol.order
    assert order(0, 4) == [0, 1, 2, 3]
    assert order(1, 4) == [2, 1, 0, 3]          # reversed, then rotated by one
    assert order(2, 4) == [2, 3, 0, 1]
    for sample in range(12):
        assert sorted(order(sample, 5)) == [0, 1, 2, 3, 4]   # every case once per sample


def test_operations_per_sample_reach_the_floor():
    bench = _bench()
    proto = bench.Protocol(torch=None)
    floor = bench.Protocol.OPS_PER_SAMPLE
    for ops in (1, 3, 4, 7, 10, 32, 33, 762):
        proto.add(f"case{ops}", lambda: None, ops)
    for name, _replay, ops, inner in proto.cases:
        assert ops * inner >= floor, name
        assert ops * (inner - 1) < floor, name       # no more graph launches than needed
    proto.add("explicit", lambda: None, 4, inner=1)
    assert proto.cases[-1][3] == 1


def test_printed_line_stays_short():
    """A reader that keeps the last 10 KB of a run's output still finds the whole line; with the rows in
    full (about 800 bytes each, 70 and more of them) it would not.  The gate reads those from stderr."""
    import json
    import xtask

    bench = _bench()
    roofline = bench.tensor_roofline("fp8_projection_kernel<128,0> splits=7 cluster-leader", 3.65e11 / 3, 1.7e8 / 3,
                                     148.12345678901234, 4500.0, 2, 6535.4)
    row = {"config": "decode", "op": "nvfp4_gate_up_swiglu_quantize", "M": 2048, "N": 16384, "K": 17408,
           "weight_copies": 12, "us": {"median": 148.12345678901234, "p10": 1.0 / 3, "p90": 2.0 / 3, "samples": 40,
                                       "operations_per_sample": 32},
           "roofline": roofline, "e2e": {"us": 1.0 / 3, "note": "x" * 80},
           "cpu_baseline": {"value": 1.0 / 3, "us_full_shape": 1e9 / 3, "sample": "x" * 160},
           "kilocycles_at_median_sm_clock": 1e3 / 3}
    assert len(json.dumps(row)) > 800
    short = [bench.line_row(row) for _ in range(75)]
    assert all(len(r) == len(bench.LINE_ROW) for r in short)
    assert len(json.dumps(short)) < 5 << 10        # the rest of the line takes about 4 KB
    rows = xtask.full_rows("a warning\n" + json.dumps({"config_row": row}) + "\n")
    line = {"config": {"rows": 1, "vocab": 248320}, "protocol": {"us_per_step": {"median": 186.0}}, "configs": rows}
    assert xtask.perf_rows(line)[("nvfp4_gate_up_swiglu_quantize", 2048, 16384)] == row["us"]["median"]
