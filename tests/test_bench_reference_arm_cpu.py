"""CPU: the benchmark's reference arm times the reference or says that it cannot.

The restatement of the transport path in oracle/ is this repository's own code: a line with "impl": "reference" must not
carry its time where the reference's source (or a host build of it) is absent.
"""
from __future__ import annotations

import json
import os
import subprocess
import sys

import pytest

import oracle_harness as H

ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")


@pytest.mark.skipif(H.reference_available(), reason="the reference is at hand")
@pytest.mark.parametrize("workload", ["small", "sweep", "surrogate"])
def test_reference_arm_without_the_reference(workload):
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--workload", workload, "--steps", "1",
                        "--warmup", "0", "--cpu-seconds", "0.1"], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
