"""bench.py's reference arm where the reference is not: it says so and times nothing in its place."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_without_the_reference(tmp_path):
    if os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libtgref.so")):
        pytest.skip("the compiled reference is here")
    env = dict(os.environ, TINY_GEMMA_REFERENCE=str(tmp_path / "none"))
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
