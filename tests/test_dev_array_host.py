"""Device arrays are complete when alloc() and upload() return
(tests/dev_array_host.cpp, host code only)."""

import shutil
import subprocess
from pathlib import Path

import pytest

from mallard_gb300 import build as B

ROOT = Path(__file__).resolve().parent.parent


def test_nothing_is_left_on_the_legacy_stream(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "dev_array"
    subprocess.run([cxx, "-std=c++20", "-O1", "-I", str(ROOT / "include"), "-I", str(B.cuda_home() / "include"),
                    str(ROOT / "tests" / "dev_array_host.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert dict(x.split("=") for x in out.split()) == {"alloc": "0", "upload": "0", "empty": "0"}
