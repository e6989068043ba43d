"""lg_exact_div.cuh against IEEE division and square root, bit for bit: random operands, significands at
the ends of their range, quotients and roots beside a rounding midpoint, extreme exponents and special
values. Correct rounding admits one result, so the tolerance is zero."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "exact_division.cu")
INC = "-I" + os.path.join(ROOT, "libgran_gb300", "csrc")


def _run(cmd, exe, arg):
    subprocess.run(cmd, check=True)
    r = subprocess.run([str(exe), str(arg)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


def test_host_build_matches_ieee(tmp_path):
    exe = tmp_path / "xd_host"
    _run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", INC, SRC, "-o", str(exe)], exe, 20000000)


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [["--fmad=false"], ["-prec-div=false", "-prec-sqrt=false", "-ftz=false"]])
def test_device_build_matches_hardware(tmp_path, flags):
    exe = tmp_path / "xd_device"
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    _run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", INC, SRC, "-o", str(exe)] + flags,
         exe, 1500)
