"""The 3-D stage's plan and the policy of its workspace, against an allocator with
a budget (host code only, compiled here): slabs cover every plane with their
halos, the limit holds, a workspace in use is not given up for one that cannot be
had, and what was refused once is not asked for again."""
from __future__ import annotations

import subprocess
from pathlib import Path

from smaug_b200.build import ARCH, CSRC, NVCC

HERE = Path(__file__).resolve().parent


def test_plan_and_workspace(tmp_path):
    exe = tmp_path / "plan3_check"
    subprocess.run([NVCC, "-std=c++17", *ARCH, "--expt-relaxed-constexpr", "-I", str(CSRC), "-o", str(exe),
                    str(HERE / "plan3_check.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
