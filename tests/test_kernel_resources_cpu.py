"""Registers of the mixed-precision kernels, as the compiler reports them (no GPU needed)."""
import os
import re
import subprocess

import __graft_entry__ as G


def _spills(source, flags, out):
    """spilled bytes (stores) of every kernel of a translation unit"""
    cmd = [G.NVCC] + G.ARCH + ["-O3", "-std=c++17", "-Xptxas", "-v", "-cubin", "-o", str(out), os.path.join(G.CSRC, source)]
    log = subprocess.run(cmd + flags, capture_output=True, text=True, check=True).stderr
    return {m.group(1): int(m.group(2))
            for m in re.finditer(r"Function properties for (\S+)\n.*?(\d+) bytes spill stores", log)}


def test_contact_kernels_do_not_spill(tmp_path):
    flags = next(f for src, _, f in G.CU_UNITS if src == "lg_forces_compact_mixed.cu")
    spills = {k: v for k, v in _spills("lg_forces_compact_mixed.cu", flags, tmp_path / "x.cubin").items() if "forces_contacts_mixed" in k}
    assert len(spills) == 3
    assert all(v <= 8 for v in spills.values()), spills  # (two registers around the loop over all pairs)
