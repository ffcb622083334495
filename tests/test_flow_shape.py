"""The flow kernels' block shape: another one would leave directions out or run past them, so it must not compile."""
import os
import subprocess

import pytest

from conftest import PKG_DIR


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_only_four_warps_compile(tmp_path, threads):
    src = tmp_path / "flow_shape.cu"
    src.write_text('#include "qcb_kernels.cuh"\n')
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-ccbin", "/usr/bin/g++",
                        "-I" + os.path.join(PKG_DIR, "csrc"), "-DQCB_FLOW_THREADS=%d" % threads, "-c", str(src),
                        "-o", str(tmp_path / "flow_shape.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == (threads == 128), r.stderr
    assert threads == 128 or "flow_map" in r.stderr
