"""Register budget of the solve kernels outside the sweeps (CPU: compiles only).

A solve kernel keeps its state in the 128 registers a thread has at 512
threads, and what does not fit is reloaded around every sweep, product and
reduction.  Where a descriptor or plan field lies is enough to change what
ptxas keeps: a pointer in the middle of SysDev and fields moved by 4 or 8
bytes raised the spills of the mixed kernel from 164 to 176 bytes and made
solves alone 0.9 to 1.2 % slower (B200); other places for the same fields
leave the fp64 or the fp16 kernel's sweeps too few registers (up to 45 %).
This test compiles the kernels with the library's own flags and `-Xptxas -v`
and holds the spilled bytes at the values they were timed with.
"""
import re
import shutil
import subprocess

import pytest

from luspice_b200 import build as b

KERNEL = "_ZN4lusp12solve_kernel{}EEvPKNS_6SysDevEiPiNS_8SmemPlanENS_11SolveParamsEiPKi{}_NS_6EscDevEi"
# (entry, spilled bytes): factor type and type of A in the inner products.
LIMITS = [(KERNEL.format("Iff", "S8"), 164), (KERNEL.format("Ifd", "S8"), 164),
          (KERNEL.format("If6__half", "S9"), 180), (KERNEL.format("Idd", "S8"), 208)]


def test_solve_kernels_spill_no_more(tmp_path):
    cmd, _ = b._cmd("cuda/engine.cu")
    if shutil.which(cmd[0]) is None:
        pytest.skip("nvcc not found")
    cmd = cmd[:-1] + [str(tmp_path / "engine.o"), "-Xptxas", "-v"]
    for name, _ in LIMITS:
        cmd += ["-Xptxas", f"--entry={name}"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = r.stderr.splitlines()
    for name, limit in LIMITS:
        at = [i for i, line in enumerate(lines) if f"Function properties for {name}" in line]
        assert len(at) == 1, name
        m = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores", lines[at[0] + 1])
        assert m and int(m.group(2)) <= limit, f"{name}: {lines[at[0] + 1].strip()}"
