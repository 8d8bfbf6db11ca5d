"""The flow sweeps' quotient with a reciprocal known beforehand against a / b, on the CPU: the function is
host-and-device code (peclet-dem_b200/csrc/pdem_flow.cuh), tests/flow_quot_check.cu compiles it for the host."""
import os
import subprocess

import pytest

import test_xadj_host as X

SRC = os.path.join(X.ROOT, "tests", "flow_quot_check.cu")
OUT = os.path.join(X.ROOT, "tests", "_build", "flow_quot_check")
CSRC = os.path.join(X.ROOT, "peclet-dem_b200", "csrc")


def test_quotient_is_correctly_rounded():
    nvcc = X._nvcc()
    if nvcc is None:
        pytest.skip("nvcc not available")
    deps = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) >= os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false",
                        "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off", "-I", CSRC, "-I",
                        os.path.join(X.ROOT, "include"), "-x", "cu", SRC, "-o", OUT], check=True, capture_output=True)
    r = subprocess.run([OUT], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]
