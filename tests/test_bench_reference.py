"""Without a build of the reference the bench's reference arm says so and times
nothing, and the CPU baseline does not go by the reference's name."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
sys.path.insert(0, ROOT)


def _without_reference():
    from oracle import oracle
    if oracle.available("ref_fast"):
        pytest.skip("a reference build is here")


def test_reference_arm_is_unavailable():
    _without_reference()
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line


def test_baseline_names_what_it_times():
    import bench
    assert bench.CPU_KINDS["reference"] == "LbmReference::Step"
    assert "restatement" in bench.CPU_KINDS["port"]
    assert 'f"LbmReference' not in open(os.path.join(ROOT, "bench.py")).read()
