"""The benchmark's reference arm measures the reference's own build or says that it cannot (no GPU)."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ORACLE, REPO


def test_reference_arm_without_the_reference_says_so():
    if os.path.exists(os.path.join(ORACLE, "_ref", "libref_emu.so")):
        pytest.skip("the reference's build is here")
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "3"], cwd=REPO,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
