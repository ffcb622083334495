"""Kernels that are launched before the launch in front of them has ended (launch_early), read in the sources.

Such a kernel runs while its inputs may still be written.  A const __restrict__ pointer, __ldg and load_ro allow
the read-only path, whose contract is that nobody writes the memory during the kernel's life.
"""
import glob
import os
import re
import subprocess

import pytest

from conftest import PKG_DIR, ROOT

CSRC = os.path.join(PKG_DIR, "csrc")
TEXT = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
        for p in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))}


def early_kernels():
    """The k_* names of every statement that calls launch_early, or that names the kernel it is given as `k`."""
    names = set()
    for text in TEXT.values():
        for m in re.finditer(r"launch_early\(\s*(\w+)", text):
            if m.group(1) == "k":
                decl = text.rfind("auto k =", 0, m.start())
                names |= set(re.findall(r"\bk_\w+", text[decl:text.index(";", decl)]))
            elif m.group(1).startswith("k_"):
                names.add(m.group(1))
    return sorted(names)


def definition(name):
    """(parameters, body) of the kernel's definition."""
    for text in TEXT.values():
        for m in re.finditer(r"\b(?:qcb::)?%s\(" % name, text):
            close = text.index(")", m.end())
            rest = text[close + 1:].lstrip()
            if not rest.startswith("{") or "__global__" not in text[max(0, m.start() - 200):m.start()]:
                continue
            depth, i = 0, text.index("{", close)
            for j in range(i, len(text)):
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                if depth == 0:
                    return text[m.end():close], text[i:j]
    raise AssertionError(name)


def test_early_kernels_are_found():
    assert {"k_finalize", "k_hb_subsweep", "k_hb_group", "k_flow_stage", "k_flow_stage1_meas", "k_meas_only",
            "k_clover_halves", "k_plaquette_planes"} <= set(early_kernels())


@pytest.mark.parametrize("name", early_kernels())
def test_early_kernel_reads_ordinary_memory(name):
    params, body = definition(name)
    assert "__restrict__" not in params
    assert "__ldg" not in body and "load_ro" not in body


@pytest.mark.gpu
def test_a_refused_launch_leaves_no_error_behind(tmp_path):
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    exe = str(tmp_path / "early_error")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-ccbin", "/usr/bin/g++",
                    "-I" + CSRC, os.path.join(ROOT, "tests", "cpp", "early_error.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
