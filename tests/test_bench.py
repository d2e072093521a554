"""The benchmark's reference arm on a machine without the reference."""
import json
import os
import subprocess
import sys

import pytest

import refharness as R

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(R.available(), reason="the reference is compiled here")
def test_reference_arm_says_that_the_reference_is_missing():
    """Nothing of this repository stands in for it: no line of figures, no library of the engine loaded."""
    code = ("import runpy, sys; sys.argv = ['bench.py', '--impl', 'reference', '--steps', '1', '--warmup', '1']; runpy.run_path('bench.py', run_name='__main__'); "
            "sys.exit(any('libvmcuda' in line for line in open('/proc/self/maps')))")
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr
    line = json.loads(done.stdout.strip())
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
