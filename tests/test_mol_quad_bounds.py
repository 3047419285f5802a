"""The half-row walk of equal molecules (molnlist.cu) reads no position beyond
the atoms: its index function, compiled for the host, over all molecule sizes
of the path, group sizes, partner counts and lanes."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_no_read_beyond_the_atoms(tmp_path):
    exe = tmp_path / "molquad_check"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", str(ROOT / "fuller_md_en_b200" / "csrc"), "-o",
                        str(exe), str(ROOT / "tests" / "cpp" / "molquad_check.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
