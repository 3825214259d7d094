"""bench.py --impl reference, which cannot run the reference here, says so in
one line and exits 0, and only on rank 0."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("rank", ["0", "1"])
def test_reference_arm_is_unavailable(rank):
    env = dict(os.environ, RANK=rank, LOCAL_RANK=rank, WORLD_SIZE="2")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "2"], cwd=ROOT,
                       env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = r.stdout.splitlines()
    if rank != "0":
        assert lines == []
        return
    line = json.loads(lines[0])
    assert len(lines) == 1 and set(line) == {"impl", "unavailable"}
    assert line["impl"] == "reference" and line["unavailable"]
