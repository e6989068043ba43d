"""Bond detection where it changes from a sweep to a hashed grid, and what degenerate shapes cost, on the CPU."""
import os
import subprocess

from libgran_gb300 import _abi as A

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_bond_paths_equal_double_loop_and_flat_shapes_stay_cheap(tmp_path):
    so = A.lib()._name
    exe = tmp_path / "bond_paths"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(ROOT, "tests", "cpp", "bond_paths.cpp"),
                    so, "-Wl,-rpath," + os.path.dirname(so), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[:2000] + r.stderr
    aggregate, chain, plane, _ = (float(v) for v in r.stdout.split())
    assert chain <= 3 * aggregate and plane <= 3 * aggregate  # (below once, measured; ten times by a sweep across them)
