"""bench.py --impl reference where the reference's library is not built: one JSON
line that says so, and exit status 0."""
from __future__ import annotations

import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("workload", ["windowed", "gxe", "biobank", "generalized"])
def test_unavailable_reference_is_one_line(workload):
    from oracle.oracle import REF_GXE_SO, REF_SO

    if (REF_GXE_SO if workload == "gxe" else REF_SO).exists():
        pytest.skip("the reference's library is built here")
    env = dict(os.environ, RANK="0")
    p = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "1",
                        "--workload", workload], capture_output=True, text=True, env=env, timeout=300)
    assert p.returncode == 0, p.stderr[-500:]
    lines = p.stdout.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["unavailable"]
