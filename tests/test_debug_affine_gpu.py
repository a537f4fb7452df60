"""The debug build's check of a sorted entry's base covers every read of the
affine rounds (tests/compat/affine_entry_check.cu, linked with the debug
library)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_entry_beyond_the_table(cuda, tmp_path):
    from liblightzk_b200 import build
    exe = str(tmp_path / "affine_entry_check")
    pkg = os.path.dirname(build.LIB_DEBUG)
    subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "-I", build.INC, "-I", build.CSRC, "--expt-relaxed-constexpr",
                    "-cudart", "shared", os.path.join(ROOT, "tests", "compat", "affine_entry_check.cu"), "-o", exe, "-L", pkg,
                    "-l:" + os.path.basename(build.LIB_DEBUG), "-Xlinker", "-rpath," + pkg, "-ccbin", "/usr/bin/g++"],
                   check=True, capture_output=True, text=True, timeout=600)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
