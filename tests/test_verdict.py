"""The word that tells a waiting host the precheck's verdict (verdict.h):
only the current solve's counts."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_a_verdict_belongs_to_its_solve(tmp_path):
    exe = tmp_path / "verdict"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-Werror", f"-I{ROOT / 'pactae_b200' / 'csrc'}",
                    str(ROOT / "tests" / "cpp" / "verdict.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and "VERDICT_OK" in out.stdout, out.stdout
