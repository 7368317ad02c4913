"""The coarse levels' one-kernel solver steps against FP64 sums, step by step.

host/step_check.cpp calls them directly, since a solve only shows a wrong coefficient
as more iterations: 1 to 16384 units of 16 bytes per right-hand side (one to eight per
thread, clusters of one to eight CTAs), 1 to 32 basis vectors.
"""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXE = os.path.join(ROOT, "grid-mg-bench_b200", "_build", "step_check")


def test_steps():
    assert os.path.exists(EXE), "build the library first (grid-mg-bench_b200/build.py)"
    r = subprocess.run([EXE], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "all steps agree" in r.stdout, r.stdout[-3000:] + r.stderr[-1000:]
