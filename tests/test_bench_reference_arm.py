"""CPU test: without the reference C the bench's reference arm says so, and measures nothing in its place."""
import json
import os
import subprocess
import sys

import pytest

import zkutil as Z


def test_reference_arm_without_the_reference_is_unavailable():
    if os.path.exists(os.path.join(Z.ROOT, "oracle", "_ref", "libzkref.so")):
        pytest.skip("the reference C is built")
    r = subprocess.run([sys.executable, os.path.join(Z.ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                        "--steps", "1", "--warmup", "1"], capture_output=True, text=True, timeout=120, cwd=Z.ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and "unavailable" in line and "value" not in line
