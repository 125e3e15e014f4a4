"""CPU test of what the engine knows of the step control without asking it
(kpolaris_b200/csrc/kp_far_steps.cuh, host build of tests/native/far_steps.cpp).

* The step-doubling error of every step of a run stays under the bound that
  macro_run takes for it.
* Every run is exactly the steps the step control takes: count, sizes and
  length, all of them in the far phase, none across the camera's radius or
  the turning point.
* The extrapolated midpoint rule lands where the steps land.  A run's RK4
  steps themselves drift from the geodesic by at most their summed
  step-doubling errors: up to 100 steps at a quarter of the tolerance 1e-6 of
  the coarsest rays would be 2.5e-5, but the bound holds at the run's inner
  end only; 1e-7 is a tenth of one step's tolerance.
* The rule itself, with the library's extrapolation, is good to 1e-11: a run
  bridged at once against the same in eight parts.
* Every step that certain_step promises to be accepted has a step-doubling
  error under half the promised one, along camera rays and for random
  vectors."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_runs_are_the_step_controls(tmp_path):
    exe = tmp_path / "far_steps"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT / 'kpolaris_b200' / 'csrc'}",
                    f"-I{ROOT / 'include'}", "-o", str(exe), str(ROOT / "tests" / "native" / "far_steps.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    const, runs, wrong, dist = float(out[0]), int(out[1]), int(out[2]), float(out[3])
    assert const <= 1.0, const
    assert runs > 1000, runs
    assert wrong == 0, wrong
    assert dist <= 1e-7, dist
    certain, worst = int(out[4]), float(out[5])
    assert certain > 100000, certain
    assert worst <= 0.5, worst
    rule, random = float(out[6]), float(out[7])
    assert rule <= 1e-11, rule
    assert random <= 0.5, random
