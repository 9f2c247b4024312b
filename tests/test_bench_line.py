"""The line that bench.py prints: one short JSON object with the headline's keys."""
import json

import bench


def test_printed_line_is_short_and_complete():
    number = 1.2345678901234567e-15
    rec = {k: number for k in ("value", "ms_per_step")}
    rec.update(
        metric=bench.METRIC, unit=bench.UNIT, n_gpus=1, steps=20, warmup=5, higher_is_better=True, scaling="weak",
        vs_baseline=None, dtype="f64 in/out; int8-valued bf16 slices on tcgen05 kind::f16, exact fp32->int accumulation",
        data="synthetic", valid=True, gpu_launches=100,
        config={"workload": bench.WORKLOAD, "l2": "x" * 80, "parallelism": "single GPU",
                **{k: 4096 for k in ("M", "N", "K", "slices", "bits", "bins", "pairs", "tile_n", "k_chunk", "stages")}},
        accuracy={"vs_exact": {"normwise_rel": number, "max_rel": number}, "vs_mpfr106": None,
                  "cublas_dgemm_vs_exact": {"normwise_rel": number}},
        elementwise_mode={"value": number, "slices": 11, "accuracy": {str(i): number for i in range(50)}},
        stage_ms={k: number for k in ("exponents", "split", "gemm", "total")},
        e2e={"value": number, "unit": bench.UNIT, "ms_per_step": number, "host_memory": "pageable (plain numpy arrays)",
             "h2d_bytes_per_step": 2 ** 28, "d2h_bytes_per_step": 2 ** 27, "pinned": {"value": number}},
        cublas_dgemm={"value": number, "unit": bench.UNIT, "ms": number},
        roofline={"bound": "tensor", "kernel": "k" * 60, "achieved": number, "peak": number, "unit": "TFLOP/s",
                  "frac": number, "traffic": {str(i): number for i in range(20)}},
        clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 1},
        cpu_baseline={"value": number, "unit": bench.UNIT, "cores": 16, "kind": "port", "sample": "s" * 100},
        sweep_4096=[{str(i): number} for i in range(400)])
    text = json.dumps(bench.contract_line(rec))
    assert len(text) < 2600 and "\n" not in text
    line = json.loads(text)
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks"):
        assert key in line, key
    assert line["accuracy"] == {"vs_exact": number, "cublas_dgemm_vs_exact": number}
