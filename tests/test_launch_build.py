"""The native call of launchers (launch.c) where it cannot be had: the kernel libraries load all the same."""

import ctypes
import glob
import os
import shutil
import subprocess
import sys

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


def test_libraries_load_where_the_module_does_not(library, folder):
    path = build._launch_path()
    if path is None:
        pytest.skip("launchers are called by ctypes here")
    with open(path, "w") as fh:
        fh.write("not a shared object")
    assert _answers(library)._native is None


def test_libraries_load_where_the_compiler_fails(library, folder, monkeypatch, capfd):
    if build._launch_path() is None:
        pytest.skip("launchers are called by ctypes here")
    (folder / "bad.c").write_text("#error no\n")
    real = build._src_path
    monkeypatch.setattr(build, "_src_path", lambda s: str(folder / "bad.c") if s == "launch.c" else real(s))
    assert _answers(library)._native is None
    said = capfd.readouterr().err
    assert "failed on launch.c" in said and "nvcc" not in said


def test_interpreters_keep_their_modules(folder, monkeypatch):
    """Two interpreters on one tree build one each, and neither removes the other's; an older source's goes."""
    if build._launch_path() is None:
        pytest.skip("launchers are called by ctypes here")
    mine = build.build_launch()
    older = mine[:-len("0123456789abcdef.so")] + "0123456789abcdef.so"
    open(older, "w").close()
    monkeypatch.setattr(sys, "version", "another interpreter")
    theirs = build.build_launch()
    assert theirs != mine and os.path.isfile(mine) and os.path.isfile(theirs) and os.path.isfile(older)
    monkeypatch.undo()
    os.environ["LITE_LANG_B200_BUILD_DIR"] = str(folder)
    try:
        os.remove(mine)
        assert build.build_launch() == mine and not os.path.isfile(older) and os.path.isfile(theirs)
    finally:
        del os.environ["LITE_LANG_B200_BUILD_DIR"]
