"""The read-outs of the recurrences by chunks: what the compiler makes of the kernel for float32 rows."""

import os
import re
import subprocess

import pytest


def test_registers_of_float32_rows():
    """Heads of 64 channels leave room for two blocks an SM (128 registers), heads of 128 do not spill (both were lost once when the
    values' address became an offset from the rows')."""
    from lite_lang_b200.csrc import build
    try:
        nvcc = build._nvcc()
    except build.BuildError:
        pytest.skip("no nvcc")
    done = subprocess.run([nvcc, *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", build._HERE, "-c",
                           build._src_path("chunk_scan.cu"), "-o", os.devnull], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr
    made = {}
    for name, stack, stores, used in re.findall(r"Compiling entry function '\w*chunk_read_kernelI(f\w*?)EEv\S*' .*?(\d+) bytes stack frame, (\d+) bytes "
                                                r"spill stores.*?Used (\d+) registers", done.stdout + done.stderr, re.S):
        made[name] = int(stores), int(used)
    assert set(made) == {"fLi64", "fLi128"}
    assert made["fLi128"][0] == 0 and made["fLi128"][1] <= 192
    assert made["fLi64"][0] <= 32 and made["fLi64"][1] <= 128
