"""The benchmark's reference arm: the reference's own kernels, or one line that says why not."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_arm_without_the_references_kernels_is_unavailable():
    from oracle.oracle import RefCpu
    if RefCpu.available():
        pytest.skip("oracle/_ref is built")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "3"], cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert r.returncode == 0 and line["impl"] == "reference" and line["unavailable"] and "value" not in line
