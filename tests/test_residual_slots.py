"""CPU: no order of the CTAs lets a residual of the resident solve be
overwritten before every CTA has read it (drot_exchange.h: residual_slot), by
exploring all orders of a 2 x 2 grid.  The model finds the fault of slots by the
iteration's parity where only even iterations are tested."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_residual_is_overwritten_unread(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "residual_slots_check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-I",
                           os.path.join(REPO, "regularized-drot_gb300", "csrc"), "-o", exe,
                           os.path.join(REPO, "tests", "native", "residual_slots_check.cpp")])
    lines = subprocess.check_output([exe], text=True).split("\n")
    found = {tuple(f[:3]): (int(f[3]), int(f[4])) for f in (t.split() for t in lines) if f}
    assert len(found) == 8
    for (rule, every, copies), (states, overwritten) in found.items():
        assert states > 1000
        if rule == "slot":
            assert overwritten == 0, (every, copies)
    assert found["parity", "0", "2"][1] > 0
    # the kernel takes its slots from that rule
    with open(os.path.join(REPO, "regularized-drot_gb300", "csrc", "drot_resident.cuh")) as f:
        uses = [t for t in f if "resx +" in t]
    assert uses and all("residual_slot(" in t for t in uses), uses
