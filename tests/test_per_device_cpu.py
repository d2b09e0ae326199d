"""What the library sets up or finds out once per device (kernel attributes,
schedulable cluster shapes): a process may have contexts on several."""
import os
import re
import subprocess

from test_device_sync_cpu import SOURCES, code

HERE = os.path.dirname(os.path.abspath(__file__))


def test_asked_once_for_each_device(tmp_path):
    exe = str(tmp_path / "per_device")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-o", exe, os.path.join(HERE, "native", "per_device.cpp")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_attribute_is_set_once_per_process():
    """cudaFuncSetAttribute holds for the current device; a once_flag or a
    static answer beside it would leave other devices without."""
    for path in SOURCES:
        src = code(path)
        assert "call_once" not in src, path
        assert not re.search(r"static std::atomic<int> ok", src), path
