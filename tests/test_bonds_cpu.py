"""Bond detection of the engine against a plain double loop, on the CPU."""
import os
import subprocess

from libgran_gb300 import _abi as A

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bond_sweep_equals_double_loop(tmp_path):
    so = A.lib()._name
    exe = tmp_path / "bond_sweep"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(ROOT, "tests", "cpp", "bond_sweep.cpp"),
                    so, "-Wl,-rpath," + os.path.dirname(so), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[:2000] + r.stderr
