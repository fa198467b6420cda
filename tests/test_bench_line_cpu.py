"""The result line of bench.py stays short: a log that keeps the last 8 KB of the output
holds all of it, however much is measured beside it."""
import json
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_result_line_is_short():
    import bench
    keys = ("metric value unit n_gpus steps warmup ms_per_step higher_is_better scaling vs_baseline dtype data "
            "iterations true_relres_max_sample roofline e2e gpu_launches clocks plain_pcg cpu_baseline").split()
    line = {k: {"text": "x" * 300} for k in keys}
    line["config"] = {"workload": "w" * 200, "launch_shapes": [[1, 256, 4, 2, 0, 120]] * 60}
    src = open(os.path.join(ROOT, "bench.py")).read()
    extras = re.findall(r'\("(\w+)", lambda:', src[src.index('for key, fn in (("single_system"'):])
    assert len(extras) >= 7
    for k in extras:  # whatever main() measures beside the result
        line[k] = {"records": ["y" * 100] * 200}
    result, detail = bench.split_line(line)
    assert len(json.dumps(result)) < 8000
    assert set(extras) <= set(detail) and not set(extras) & set(result)
    assert set(keys) <= set(result) and result["config"] == {"workload": "w" * 200}
    assert line["config"]["launch_shapes"] == detail["launch_shapes"]
