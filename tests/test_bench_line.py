"""The line that the benchmark prints: one JSON object on stdout, short, with every required key; details on stderr.  The
reference arm times the oracle and loads nothing of the package."""
import json
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_line_is_short_and_keeps_what_is_required(capsys):
    sys.path.insert(0, str(ROOT))
    import bench_common as bc

    line = {"metric": "m", "value": 1 / 3, "config": {"workload": "w" * 400}, "e2e": {"value": 2 / 3, "h2d_bytes_per_step": 536870912},
            "clocks": {"sm_mhz": 1.0}, "roofline": {"frac": 0.5}, "extras": {str(i): 1 / 7 for i in range(400)}}
    details = {"shapes": {str(i): {"ms": 1 / 7} for i in range(400)}}
    bc.print_line(line, details)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 2700
    got = json.loads(out)
    assert "extras" not in got and got["value"] == 0.333333 and got["e2e"]["h2d_bytes_per_step"] == 536870912
    assert json.loads(err) == {**line, **details}
    bc.print_line({"metric": "m", "extras": {"a": 1}})
    out, err = capsys.readouterr()
    assert json.loads(out) == {"metric": "m", "extras": {"a": 1}} and err == ""


def test_reference_arm_loads_nothing_of_the_package():
    code = ("import sys, bench_stack, oracle\n"
            "class A: workload, layers, attention = 'tp_stack', 0, 'identity'\n"
            "tp, cfg, (batch, seq), seed = bench_stack._config(A)\n"
            "assert bench_stack.workload_string(cfg, batch, seq) and cfg.q_width == 8192 and cfg.kv_width == 1024\n"
            "assert not [m for m in sys.modules if m.startswith('tensorrt_b200')]\n")
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True, timeout=300)


def test_shapes_are_those_of_the_package():
    import dataclasses

    sys.path.insert(0, str(ROOT))
    import bench_stack
    from tensorrt_b200.stack import LLAMA3_8B, LLAMA3_70B, StackConfig

    assert StackConfig(**dataclasses.asdict(bench_stack.SHAPES["tp_stack"])) == LLAMA3_70B
    assert StackConfig(**dataclasses.asdict(bench_stack.SHAPES["nvfp4_stack"])) == LLAMA3_8B
