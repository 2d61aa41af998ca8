"""The bench's result line: one JSON object on stdout with the contract's keys,
short enough for a log's tail; the details go to stderr."""

import argparse
import json

import bench

CONTRACT = {"metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
            "vs_baseline", "dtype", "data", "config", "clocks", "e2e", "gpu_launches"}


def test_result_line(capsys):
    args = argparse.Namespace(probe_s=0.0, steps=20, refine=4, slots=8, max_batch=64, batch_pixels=512 * 512,
                              linger_us=0, records="half_normals", arithmetic="fast", serving_volumes=32,
                              serving_extra=224, gpus=1)
    result = {k: 1234.567890123456 for k in bench.HEADLINE_KEYS}
    result.update(metric="renders/s (batched server, mixed request stream, p99 of 512^2 frames <= 20 ms)",
                  config=bench.serving_config(args), clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
                  e2e={"value": 1234.567890123456, "unit": "renders/s", "h2d_bytes_per_step": 123456789.0123,
                       "d2h_bytes_per_step": 123456789.0123},
                  cpu_baseline={"sample": "x" * 500}, serial_per_frame={"renders_per_s": 1.0, "p50_ms": 1.0})
    details = {"plain": {"x": ["y"] * 5000}, "probes": {"server": [{"n": 1}] * 1000}}
    bench.print_result({**details, **result})
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 4096
    line = json.loads(out)
    assert line == result and CONTRACT <= set(line)
    assert json.loads(err) == details
