"""CPU test of the mixed policy's thermal-synchrotron fits
(kpolaris_b200/csrc/kp_radiation_mixed.cuh, built for the host from
tests/native/mixed_coefficients.cpp) against the reference's FP64 values stored
in tests/golden/coefficients.npz.

Tolerance: 1e-9 relative per coefficient.  The fits are the reference's with
their factors regrouped and powers taken through logarithms; what costs digits
is a logarithm or root of relative error e under an exponential of argument a,
a e: 1e-16 times the at most 1e3 of a significant coefficient, and 1e-12 of the
Newton cube root under exp(-x^(1/3)).  Single precision anywhere would be off
by 1e-7."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "native" / "mixed_coefficients.cpp"


@pytest.fixture(scope="module")
def binary(tmp_path_factory):
    exe = tmp_path_factory.mktemp("mixed") / "mixed_coefficients"
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{ROOT / 'kpolaris_b200' / 'csrc'}", f"-I{ROOT / 'include'}",
                    "-o", str(exe), str(SRC)], check=True)
    return exe


def test_mixed_fits_match_reference(binary):
    fx = np.load(ROOT / "tests" / "golden" / "coefficients.npz")
    pts = fx["thermal_in"]
    want = fx["thermal_out"]
    text = "\n".join(" ".join(f"{v:.17g}" if i else str(int(v)) for i, v in enumerate(p)) for p in pts)
    out = subprocess.run([str(binary)], input=text, capture_output=True, text=True, check=True).stdout
    got = np.array([[float(v) for v in line.split()] for line in out.strip().splitlines()])
    # columns: jI jQ jV aI aQ aV rQ rV  <->  reference indices 0 1 3 4 5 7 8 10
    ref = want[:, [0, 1, 3, 4, 5, 7, 8, 10]]
    assert got.shape == ref.shape
    scale = np.maximum(np.abs(ref), 1e-300)
    rel = np.abs(got - ref) / scale
    # what is 30 decades under a coefficient's largest value is exempt
    significant = np.abs(ref) > 1e-30 * np.max(np.abs(ref), axis=0)
    assert np.all(rel[significant] <= 1e-9), rel[significant].max()
