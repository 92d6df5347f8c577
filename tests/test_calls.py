"""The call extension: arguments as the functions' signatures say, on a small library of its own."""

import ctypes
import shutil
import subprocess

import pytest

from acorninfer_b200.kernels import calls

SOURCE = """
extern "C" long long mix(void* p, int a, long long b, float c, void* q) { return (long long)(unsigned long long)p + 10 * a + b + (long long)(4 * c) + (q == nullptr); }
extern "C" int none() { return -7; }
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_calls_convert_and_refuse_arguments(tmp_path):
    src, lib = tmp_path / "small.cpp", tmp_path / "libsmall.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-shared", "-fPIC", str(src), "-o", str(lib)], check=True)
    signatures = {"mix": ([ctypes.c_void_p, ctypes.c_int, ctypes.c_int64, ctypes.c_float, ctypes.c_void_p], ctypes.c_int64),
                  "none": ([], ctypes.c_int)}
    loaded = ctypes.CDLL(str(lib))
    fns = calls.load(signatures, lib, tmp_path)
    if not fns:
        pytest.skip("no Python headers")
    assert loaded.none() == -7 == fns["none"]()
    assert fns["mix"](1 << 40, -3, 1 << 41, 0.25, None) == (1 << 40) - 30 + (1 << 41) + 1 + 1
    assert fns["mix"](None, True, -1, 2, 8) == 10 - 1 + 8
    for bad, error in (((None, 1, 1, 1.0), TypeError), ((None, 1 << 31, 1, 1.0, None), OverflowError), ((1.5, 1, 1, 1.0, None), TypeError),
                       ((None, 1, 1 << 63, 1.0, None), OverflowError), ((None, 1, 1, "x", None), TypeError)):
        with pytest.raises(error):
            fns["mix"](*bad)
    assert calls.load(signatures, lib, tmp_path)["none"]() == -7          # built once
    with pytest.raises(RuntimeError):
        calls.load({"other": ([], ctypes.c_int)}, lib, tmp_path)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_a_compiler_or_an_import_that_fails_leaves_the_calls_to_ctypes(tmp_path, monkeypatch):
    src, lib = tmp_path / "small.cpp", tmp_path / "libsmall.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-shared", "-fPIC", str(src), "-o", str(lib)], check=True)
    signatures = {"none": ([], ctypes.c_int)}
    loaded = ctypes.CDLL(str(lib))
    path = calls.build(signatures, tmp_path)
    if path is None:
        pytest.skip("no Python headers")
    path.write_bytes(b"not an extension")
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert calls.load(signatures, lib, tmp_path) == {}
    path.unlink()
    tools = tmp_path / "tools"
    tools.mkdir()
    (tools / "g++").write_text("#!/bin/sh\necho unknown standard c++17 >&2\nexit 1\n")
    (tools / "g++").chmod(0o755)
    monkeypatch.setenv("PATH", str(tools), prepend=":")
    with pytest.warns(RuntimeWarning, match="unknown standard"):
        assert calls.load(signatures, lib, tmp_path) == {}
    with pytest.raises(RuntimeError):               # the build step itself says so
        calls.build(signatures, tmp_path)
    assert loaded.none() == -7 and not list(tmp_path.glob("acorn_calls*"))


def test_a_given_library_keeps_its_folder(tmp_path, monkeypatch):
    from acorninfer_b200.kernels import build
    given, own = tmp_path / "given", tmp_path / "own"
    given.mkdir()
    lib = given / "lib.so"
    lib.write_bytes(b"")
    monkeypatch.delenv("ACORN_KERNEL_LIB", raising=False)
    monkeypatch.setenv("ACORN_BUILD_DIR", str(own))
    assert build.own_folder(lib) == given
    monkeypatch.setenv("ACORN_KERNEL_LIB", str(lib))
    assert build.own_folder(build.ensure_built()) == own and own.is_dir() and list(given.iterdir()) == [lib]
