"""bench.py's reference arm: without the compiled reference it says so in one line and exits 0, and
never reports another program's time under the reference's name."""
import json
import os
import subprocess
import sys

import pytest

from oracle import ref
from tests.helpers import ROOT


@pytest.mark.skipif(ref.available("tim"), reason="the compiled reference is here")
def test_unavailable_line():
    env = {**os.environ, "OMP_NUM_THREADS": "1"}
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "1",
                        "--steps", "2", "--warmup", "3"], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
