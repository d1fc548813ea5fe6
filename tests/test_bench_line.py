"""What the benchmark's line says about a step's bound, and its reference arm."""

import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("n,pml,eps,in_place,bound,fields", [
    (128, 10, True, True, "l2", 76.0),    # 70 MB of fields and psi
    (64, 8, False, True, "l2", 72.0),
    (256, 12, True, True, "hbm", 76.0),   # 0.5 GB
    (128, 10, True, False, "hbm", 52.0),  # two buffer sets, one pass
    (512, 12, True, False, "hbm", 52.0),
])
def test_step_roofline(n, pml, eps, in_place, bound, fields):
    import bench

    got = bench.step_roofline(n, pml, eps, in_place)
    assert got == (bound, fields + bench.psi_bytes_per_cell(n, pml))


def test_reference_arm_reports_itself_unavailable():
    """It runs the reference or nothing: never this repository's own restatement."""
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps",
                          "1", "--warmup", "3"], capture_output=True, text=True, check=True,
                         timeout=300).stdout
    line = json.loads(out)
    assert line["impl"] == "reference" and "JAX" in line["unavailable"] and "value" not in line
