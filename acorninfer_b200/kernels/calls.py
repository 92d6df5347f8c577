"""Calls into the kernel library without ctypes' conversions.

A call of 25 to 40 arguments costs ctypes 3 to 4 us, as much as the launch behind it: a step of a few hundred tokens that is not
replayed from a graph makes 100 to 300 of them and is bound by the host.  ``load`` makes a small extension module from the
functions' signatures (one typed call each, compiled with the Python headers) and returns its functions by name; an
argument costs 5 to 10 ns there.  Without those headers or a C++ compiler, or where the compiler or the import fails (which a warning
says), it returns nothing and ctypes does the calls.
Steps of 27 decoded rows and 3 prompts at Qwen3-0.6B sizes: 4.83 -> 4.29 ms; three prompts of a design with 185 launches 3.15 -> 2.91 ms.
"""

from __future__ import annotations

import ctypes
import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import warnings
from pathlib import Path

_TYPES = {ctypes.c_void_p: "void*", ctypes.c_int: "int", ctypes.c_int64: "long long", ctypes.c_float: "float"}

_HEAD = """// Typed calls of the kernel library's functions (generated from their signatures).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>
#include <tuple>

static bool take(PyObject* o, void** v) { return o == Py_None ? (*v = nullptr, true) : (*v = PyLong_AsVoidPtr(o), *v != nullptr || !PyErr_Occurred()); }
static bool take(PyObject* o, long long* v) { *v = PyLong_AsLongLong(o); return *v != -1 || !PyErr_Occurred(); }
static bool take(PyObject* o, float* v) { const double d = PyFloat_AsDouble(o); *v = (float)d; return d != -1.0 || !PyErr_Occurred(); }
static bool take(PyObject* o, int* v) {
    const long l = PyLong_AsLong(o);
    if (l == -1 && PyErr_Occurred()) return false;
    *v = (int)l;
    if (*v != l) { PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits"); return false; }
    return true;
}

static void* fns[COUNT];

template <int I, typename R, typename... A>
static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != (Py_ssize_t)sizeof...(A)) return PyErr_Format(PyExc_TypeError, "%zd arguments given, %zd taken", n, (Py_ssize_t)sizeof...(A));
    std::tuple<A...> t;
    const bool ok = std::apply([&](auto&... v) { PyObject* const* p = args; (void)p; return (take(*p++, &v) && ... && true); }, t);
    if (!ok) return nullptr;
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = std::apply(reinterpret_cast<R (*)(A...)>(fns[I]), t);
    Py_END_ALLOW_THREADS
    return PyLong_FromLongLong((long long)r);
}
"""

_TAIL = """
// Looks the functions up in the library at `path`, which the process has loaded.
static PyObject* bind(PyObject*, PyObject* path) {
    const char* name = PyUnicode_AsUTF8(path);
    if (name == nullptr) return nullptr;
    void* lib = dlopen(name, RTLD_NOW | RTLD_NOLOAD);
    if (lib == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s is not loaded", name);
    for (int i = 0; i < COUNT; ++i) {
        fns[i] = dlsym(lib, methods[i].ml_name);
        if (fns[i] == nullptr) return PyErr_Format(PyExc_RuntimeError, "%s lacks %s", name, methods[i].ml_name);
    }
    Py_RETURN_NONE;
}
"""


def source(signatures: dict[str, tuple[list, object]]) -> str:
    """The extension's C++ source: ``signatures`` maps a function's name to its ctypes argument and result types."""
    rows = [f'    {{"{name}", (PyCFunction)(void (*)())call<{i}, {_TYPES[result]}{"".join(", " + _TYPES[a] for a in args)}>, METH_FASTCALL, nullptr}},'
            for i, (name, (args, result)) in enumerate(sorted(signatures.items()))]
    return (f"#define COUNT {len(rows)}\n" + _HEAD + "\nstatic PyObject* bind(PyObject*, PyObject*);\nstatic PyMethodDef methods[] = {\n"
            + "\n".join(rows) + '\n    {"bind", bind, METH_O, nullptr},\n    {nullptr, nullptr, 0, nullptr}};\n' + _TAIL
            + '\nstatic PyModuleDef module = {PyModuleDef_HEAD_INIT, "acorn_calls", nullptr, -1, methods};\n'
            "PyMODINIT_FUNC PyInit_acorn_calls() { return PyModule_Create(&module); }\n")


def build(signatures: dict[str, tuple[list, object]], folder: Path) -> Path | None:
    """Compiles the extension into ``folder`` if it is not there yet; None without a compiler, headers or a folder that can be
    written; a compiler that fails raises."""
    text, suffix = source(signatures), sysconfig.get_config_var("EXT_SUFFIX")
    include, gxx = sysconfig.get_paths()["include"], shutil.which("g++")
    digest = hashlib.sha256((text + sys.version).encode()).hexdigest()[:16]
    target = folder / f"acorn_calls_{digest}{suffix}"
    if target.is_file():
        return target
    if gxx is None or not (Path(include) / "Python.h").is_file():
        return None
    src, tmp = folder / f"acorn_calls_{digest}.{os.getpid()}.cpp", folder / f"acorn_calls_{digest}.tmp{os.getpid()}"
    try:
        src.write_text(text)
        res = subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", include, str(src), "-o", str(tmp), "-ldl"],
                             capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"g++ failed on the call extension:\n{res.stderr}")
        os.replace(tmp, target)
    except OSError:                     # a folder that cannot be written
        return None
    finally:
        for left in (src, tmp):
            try:
                left.unlink()
            except OSError:
                pass
    return target


def load(signatures: dict[str, tuple[list, object]], library: Path, folder: Path) -> dict[str, object]:
    """The library's functions by name as the extension calls them (``library`` is loaded); empty where it cannot be built or
    imported."""
    try:
        path = build(signatures, folder)
        if path is None:
            return {}
        spec = importlib.util.spec_from_file_location("acorn_calls", path)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
    except (RuntimeError, ImportError, OSError) as e:
        warnings.warn(f"kernels are called through ctypes, which is slower: no call extension ({e})", RuntimeWarning, stacklevel=2)
        return {}
    module.bind(str(library))
    return {name: getattr(module, name) for name in signatures}
