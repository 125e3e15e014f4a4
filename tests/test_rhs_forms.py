"""CPU check of the mixed policy's factored transport right-hand sides (host
build of tests/native/rhs_forms.cpp) against the reference-order FP64 ones on
20000 seeded states: Kerr-Schild (kpolaris_b200/csrc/kp_geometry_mixed.cuh) and
FMKS (kpolaris_b200/csrc/kp_fmks.cuh) within 1e-12 normwise (they regroup the
same algebra)."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_factored_rhs_matches_reference_order(tmp_path):
    exe = tmp_path / "rhs_forms"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'kpolaris_b200' / 'csrc'}",
                    f"-I{ROOT / 'include'}", "-o", str(exe), str(ROOT / "tests" / "native" / "rhs_forms.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    for form, worst in zip(("Kerr-Schild", "FMKS"), out):
        assert float(worst) <= 1e-12, (form, worst)
