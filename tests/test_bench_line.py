"""bench.py's result line: one JSON line on stdout, short enough for a reader that
keeps only the end of the output; the legs beside it go to stderr."""
import json

import bench


def test_result_line_is_short_and_alone(capsys):
    row = {"N": 1024, "window": "hamming", "output": "half_complex", "gsamples_s": 123.45, "ms": 1.2345,
           "hbm_frac": 0.987, "fp32_pipe": {"gflop_s": 12345.6, "peak_gflop_s": 80546.4, "frac": 0.1234}}
    contract = {"metric": "Gsamples/s", "value": 1.0, "unit": "Gsamples/s", "n_gpus": 1, "steps": 1, "warmup": 3,
                "ms_per_step": 0.2, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic", "config": {"workload": "w" * 300}, "roofline": {"frac": 0.9},
                "e2e": {"value": 1.0, "unit": "Gsamples/s"}, "gpu_launches": 1, "clocks": {"sm_mhz": 2070.0},
                "accuracy": {"rel_l2": 1e-7}, "cpu_baseline": {"value": 0.1, "sample": "s" * 300}}
    legs = {"sweep": [row] * 68, "cufft_reference": {"a": 1}, "tensor_core": [row] * 20, "uneven_batch": {"a": 1},
            "serving": {"rates": [row] * 5}, "runner_executable": {"a": 1}}
    bench.report({**contract, **legs})
    out = capsys.readouterr()
    assert json.loads(out.out) == contract and out.out.count("\n") == 1
    assert len(out.out) < 4096
    assert json.loads(out.err.split("bench legs: ", 1)[1]) == legs
