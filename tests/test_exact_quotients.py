"""The FP64 policy's quotients and square roots (kpolaris_b200/csrc/kp_exact.cuh)
are IEEE's, bit for bit: exact_quots and KP_OVER for any operands, exact_recip,
exact_quot and exact_sqrt within the ranges they state.

The operands (tests/native/exact_quotients.h) cover both signs, zeros of both
signs, subnormal numbers, infinities and NaN, the ends of the admitted ranges
and just beyond them, and significands of all ones, nearly so, and powers of
two.

* CPU: tests/native/exact_quotients.cpp, the method with C's fma and
  starting values of 20 bits, exact but for them and off by twice as much.
* GPU: tests/native/exact_quotients.cu, against CUDA's own operators.

The mixed policy's reciprocals and roots (kp_geometry_mixed.cuh,
kp_radiation_mixed.cuh) are not exact.  On the GPU: kp_recip and kp_sqrt_pair
within 4 ulp, cube_root within 1e-12 for x in 1..1e7 and 1e-11 beyond -- a
single-precision root is off by at most log(x) 2^-23 / 3, and Newton's step
squares that."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NATIVE = ROOT / "tests" / "native"
CSRC = ROOT / "kpolaris_b200" / "csrc"


@pytest.mark.parametrize("err", [0.0, 2e-6])
def test_host_emulation(tmp_path, err):
    exe = tmp_path / "exact_quotients"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}", f"-I{ROOT / 'include'}", f"-I{NATIVE}",
                    "-o", str(exe), str(NATIVE / "exact_quotients.cpp")], check=True)
    out = subprocess.run([str(exe), "2000000", repr(err)], capture_output=True, text=True, check=True).stdout.split()
    assert [int(x) for x in out] == [0] * 5, dict(zip(("quots", "over", "quot", "recip", "root"), out))


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    so = tmp_path_factory.mktemp("exact") / "exact_quotients.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "--fmad=false",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", f"-I{CSRC}", f"-I{ROOT / 'include'}", f"-I{NATIVE}",
                    "-shared", "-o", str(so), str(NATIVE / "exact_quotients.cu")], check=True)
    return C.CDLL(str(so))


@pytest.mark.gpu
def test_device_operators(device):
    counts = (C.c_ulonglong * 5)()
    rc = device.kp_probe_exact_quotients(400, counts)
    assert rc == 0, f"cudaError {rc}"
    assert list(counts) == [0] * 5, dict(zip(("quots", "over", "quot", "recip", "root"), counts))


@pytest.mark.gpu
def test_device_mixed_roots(device):
    errors = (C.c_double * 5)()
    rc = device.kp_probe_mixed_roots(400, errors)
    assert rc == 0, f"cudaError {rc}"
    ulp = 2.0 ** -52
    assert all(e <= bar for e, bar in zip(errors, (4 * ulp, 4 * ulp, 4 * ulp, 1e-12, 1e-11))), list(errors)
