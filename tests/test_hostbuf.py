"""The host buffers that the server uses again, in a plain C++ program."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_host_buffers(tmp_path):
    exe = str(tmp_path / "hostbuf_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-pthread", "-I" + os.path.join(PKG_DIR, "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "hostbuf_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
