"""CPU check of the rules that choose a solve's kernel (csrc/route.h), compiled with g++."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_routes(tmp_path):
    exe = tmp_path / "route_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(ROOT / "capellinisptrsv_gb300" / "csrc"),
                    str(ROOT / "tests" / "native" / "route_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "routes ok" in r.stdout
