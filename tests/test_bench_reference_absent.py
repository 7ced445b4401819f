"""The benchmark's CPU baseline where the reference is not built: its worker's
error reaches the caller (a pool waits for good on one that it cannot unpickle)."""
import subprocess
import sys
from pathlib import Path

import pytest

import oracle_bind as ob

ROOT = Path(__file__).resolve().parents[1]
RUN = """
import sys
sys.path.insert(0, {root!r})
import bench
if __name__ == "__main__":
    try:
        bench.cpu_reference_rate(1, 16, 1)
    except OSError as e:
        print("not built:", type(e).__module__, e.filename)
"""


@pytest.mark.skipif(ob.REF_PERF.exists() or ob.REFERENCE_TREE is not None, reason="the reference is built here")
def test_the_workers_error_reaches_the_caller(tmp_path):
    f = tmp_path / "run.py"
    f.write_text(RUN.format(root=str(ROOT)))
    r = subprocess.run([sys.executable, str(f)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.strip() == f"not built: builtins {ob.REF_PERF}"
