"""The reference arm of bench.py where the reference can be neither found nor
built: one JSON line that says so, and status 0 (CPU only)."""
import json
import os
import subprocess
import sys

import pytest

from oracle import ref

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(ref.available(), reason="the reference library is built")
@pytest.mark.parametrize("sources", ["absent", "empty"])
@pytest.mark.parametrize("args", [(), ("--workload", "batched512"), ("--workload", "wells256"),
                                  ("--workload", "peierls2048")])
def test_reference_arm_without_the_reference(tmp_path, sources, args):
    where = tmp_path / "reference"
    if sources == "empty":
        where.mkdir()
    p = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1",
                        "--warmup", "3", *args], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, TRLAN_REFERENCE=str(where)))
    assert p.returncode == 0, p.stderr[-2000:]
    line, = [json.loads(x) for x in p.stdout.splitlines() if x.startswith("{")]
    assert line["impl"] == "reference" and str(where) in line["unavailable"]
