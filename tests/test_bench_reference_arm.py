"""bench.py's reference arm (the reference CPU filter, restated by the
oracle, timed on the host's cores) needs no GPU: it prints one JSON line
with the base contract's keys, and under torchrun only rank 0 prints it."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(extra_env=None):
    env = dict(os.environ)
    env.update(extra_env or {})
    return subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3"],
                          cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)


def test_reference_arm_line():
    r = _run()
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference"
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "higher_is_better", "config",
                "cpu_baseline", "e2e"):
        assert key in line, key
    assert line["value"] > 0 and line["higher_is_better"] is True
    assert line["config"]["workload"] == "l96_d40_n65536"
    cb = line["cpu_baseline"]
    assert cb["kind"] in ("port", "reference") and cb["cores"] >= 1 and cb["sample"]
    assert cb["value"] == line["value"]
    assert line["e2e"]["value"] == line["value"]
    assert line["e2e"]["h2d_bytes_per_step"] == 0 and line["e2e"]["d2h_bytes_per_step"] == 0


def test_reference_arm_other_ranks_print_nothing():
    r = _run({"RANK": "1", "WORLD_SIZE": "2", "LOCAL_RANK": "1"})
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == ""


def test_own_arm_line_is_short():
    """The line on standard output holds the contract's keys and names the
    sections that went to standard error."""
    sys.path.insert(0, ROOT)
    import bench

    line = {"metric": bench.METRIC, "value": 1.0, "e2e": {"value": 1.0}, "clocks": {}, "cpu_baseline": {"value": 1.0}}
    sections = {k: {"x": "y" * 20000} for k in bench.DETAIL}
    line.update(sections)
    assert bench.split_detail(line) == sections
    assert line["detail"] == sorted(bench.DETAIL)
    assert set(line) == {"metric", "value", "e2e", "clocks", "cpu_baseline", "detail"}
    headline = {"metric": bench.METRIC, "value": 1.0}
    assert bench.split_detail(headline) == {} and "detail" not in headline
