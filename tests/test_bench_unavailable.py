"""bench.py's reference arm on a machine without the reference's kernels: a step that the host
cannot compute whole is `unavailable`, not the restatement's extrapolation under its name."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_large_step_is_unavailable():
    import refslice
    if refslice.available():
        pytest.skip("the reference's kernels are built here")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1"],
                       capture_output=True, text=True, env=dict(os.environ, RANK="0"), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [json.loads(l) for l in r.stdout.splitlines() if l.strip()]
    assert len(lines) == 1 and set(lines[0]) == {"impl", "unavailable"} and lines[0]["impl"] == "reference"
    assert lines[0]["unavailable"] and "\n" not in lines[0]["unavailable"]
