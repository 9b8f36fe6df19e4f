"""Host check of the stack that a team of lanes shares (no GPU).

`tests/cpp/team_stack_check.cpp` runs the stack step of the team traversal
(`devilray_gb300/csrc/team_stack.cuh`) with the lanes as threads that take turns
in a given order between two barriers, and compares the nodes that every lane
visits with a walk of its own: a pop and a push of the same entry that no barrier
separates shows as soon as the writing lane runs first.
"""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA_INCLUDE = Path("/usr/local/cuda/include")


def test_team_lanes_agree_in_any_order(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    exe = tmp_path / "team_stack_check"
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", str(ROOT / "devilray_gb300" / "csrc"), "-I", str(CUDA_INCLUDE),
                    str(ROOT / "tests" / "cpp" / "team_stack_check.cpp"), "-o", str(exe), "-pthread"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    assert words[0] == "ok" and int(words[1]) > 1000
