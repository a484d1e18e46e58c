"""Kernel attributes are set once on every device, not once per process."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "impec2d_gb300", "csrc")


def test_once_per_device(tmp_path):
    exe = tmp_path / "once"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", os.path.join(ROOT, "tests", "cpp", "once_per_device.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_launchers_set_limits_per_device():
    """A launcher that sets a kernel's shared-memory limit does so through allow_smem; contexts set theirs each time
    one is created (pressure.cu).  No flag for the whole process decides it."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r"static\s+bool\s+attr", text), name
            if name not in ("pressure.cu", "internal.cuh"):
                assert "cudaFuncSetAttribute" not in text, name
