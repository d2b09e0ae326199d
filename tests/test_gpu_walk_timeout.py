"""A block walk (blockwalk.cu) given up because a wait ran out: it ends, within
its arrays, is reported, and leaves the context and the next walk sound."""
import os
import subprocess

import pytest

from ressim_gb300 import build

pytestmark = pytest.mark.gpu


def test_walk_given_up(tmp_path):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "block_walk_timeout.cu")
    exe = str(tmp_path / "block_walk_timeout")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-o", exe, src, "-L" + build.LIB_DIR, "-lresgpu",
                    "-Xlinker", "-rpath", "-Xlinker", build.LIB_DIR], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("ended\n"), r.stdout + r.stderr
