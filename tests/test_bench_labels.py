"""The reference arm says what ran: the reference's own functions, or the port of this repository where those were not built."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT


@pytest.mark.parametrize("fmt", ["q4", "nvfp4"])
def test_sample_names_what_ran(fmt):
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0",
                          "--layers", "1", "--format", fmt], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout)["cpu_baseline"]
    assert ("own functions" in line["sample"]) == (line["kind"] == "reference")
    assert ("CPU port" in line["sample"]) == (line["kind"] == "port")
