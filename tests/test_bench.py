"""bench.py's reference arm without a GPU: a measured line, or a line that
says why there is none."""
import json
import subprocess
import sys
from pathlib import Path

import oracle

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_measures_or_says_why_not():
    res = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--scale", "10",
                          "--steps", "1", "--warmup", "0"], capture_output=True, text=True,
                         timeout=300, cwd=ROOT)
    assert res.returncode == 0 and "Traceback" not in res.stderr, res.stderr[-2000:]
    line = json.loads(res.stdout)
    assert line["impl"] == "reference"
    if oracle.have_reference():
        assert line["value"] > 0 and "unavailable" not in line
    else:
        assert line["unavailable"] and "value" not in line
