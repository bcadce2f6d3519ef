"""The cache of freed device blocks (strobealign_gb300/csrc/devcache.h) over a fake device
with two devices and three contexts (CPU, compiled with g++)."""
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_blocks_of_several_places(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", f"-I{ROOT / 'strobealign_gb300' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "device_cache_check.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
