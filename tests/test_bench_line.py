"""bench.py prints one line that a reader with a small buffer can take in: the served
window's per-job records go to a file of their own."""
import json
import os
import subprocess
import sys

import bench


def line(jobs):
    rep = {"jobs": jobs, "latency_p50_s": 1.0,
           "job_records": [{"job": k, "dim": 2, "n": 5776, "steps": 3348, "arrival": 8.5 + k,
                            "finished": 53.9 + k, "error": None} for k in range(jobs)]}
    return {"metric": bench.METRIC, "value": 1.0, "unit": bench.UNIT,
            "workloads": {"batched": {"sims": 512, "value": 2.0}, "serve": rep}}


def test_line_does_not_grow_with_the_jobs(tmp_path):
    few, many = bench.result_line(line(2)), bench.result_line(line(2000))
    assert len(many) - len(few) < 200
    got = json.loads(many)
    assert got["value"] == 1.0 and got["workloads"]["batched"]["sims"] == 512
    assert "job_records" not in got["workloads"]["serve"]
    assert got["workloads"]["serve"]["jobs"] == 2000


def test_records_go_to_a_file(tmp_path):
    path = tmp_path / "details.json"
    bench.result_line(line(5), str(path))
    assert [r["job"] for r in json.loads(path.read_text())["job_records"]] == list(range(5))
    bench.result_line({"metric": bench.METRIC, "value": 1.0}, str(path))


def test_reference_arm_says_that_there_is_none():
    """Nothing of this repository is timed in the reference's name."""
    path = os.path.join(bench.ROOT, "bench.py")
    res = subprocess.run([sys.executable, path, "--impl", "reference", "--steps", "2"],
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    got = json.loads(res.stdout)
    assert got["impl"] == "reference" and got["unavailable"] and "value" not in got
