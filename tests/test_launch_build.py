"""The native call of launchers (launch.c) where it cannot be had: the kernel libraries load all the same."""

import ctypes
import glob
import os
import shutil
import subprocess

import pytest

from lite_lang_b200.csrc import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def library(tmp_path):
    """A launcher without a GPU: the sum of its two parameters, as its error code."""
    cc = shutil.which("cc") or shutil.which("gcc")
    if cc is None:
        pytest.skip("no host compiler")
    source, path = tmp_path / "sum.c", str(tmp_path / "sum.so")
    source.write_text("int sum(int a, long b) { return a + (int)b; }\n")
    subprocess.run([cc, "-shared", "-fPIC", str(source), "-o", path], check=True)
    return path


@pytest.fixture
def folder(tmp_path, monkeypatch):
    monkeypatch.setenv("LITE_LANG_B200_BUILD_DIR", str(tmp_path / "built"))
    return tmp_path / "built"


def _answers(path):
    lib = build.Library("sum", path)
    lib.call("sum", 3, -3)
    with pytest.raises(RuntimeError, match="CUDA error 7"):
        lib.call("sum", 3, ctypes.c_long(4))
    return lib


def test_a_package_has_every_source():
    """What an installed package's folder of sources holds is what the build of its libraries reads."""
    import setuptools
    seen, real = {}, setuptools.setup
    setuptools.setup = lambda **kw: seen.update(kw)
    here = os.getcwd()
    try:
        os.chdir(ROOT)
        exec(compile(open("setup.py").read(), "setup.py", "exec"), {})
    finally:
        os.chdir(here)
        setuptools.setup = real
    folder = os.path.dirname(os.path.abspath(build.__file__))
    shipped = {p for pattern in seen["package_data"]["lite_lang_b200.csrc"] for p in glob.glob(os.path.join(folder, pattern))}
    read = {p for sources, _ in build.LIBRARIES.values() for p in build._with_includes(sources)} | {build._src_path("launch.c")}
    assert {os.path.abspath(p) for p in read} <= shipped


def test_libraries_load_without_the_source(library, folder, monkeypatch):
    real = build._src_path
    monkeypatch.setattr(build, "_src_path", lambda s: str(folder / "none.c") if s == "launch.c" else real(s))
    assert build.build_launch() is None and _answers(library)._native is None
