"""Builds and loads the CUDA extension (the ``.cu`` files under ``csrc/``).

The extension is one shared library of ``extern "C"`` launchers, compiled with ``nvcc`` for
sm_100a; launchers take raw device pointers and a stream.  Python calls them through wrappers that are
made from their prototypes and compiled into the same library (:func:`launchers`): a call of twenty arguments
through ``ctypes`` costs as much as the launch it makes.  The library is built
in-tree (``lalamo_b200/_native/``) when that folder can be written, otherwise under the
temporary directory, and rebuilt when a source file changes.  There is no fallback: if the
library cannot be built or loaded, :func:`library` raises.
"""

from __future__ import annotations

import ctypes
import hashlib
import importlib.machinery
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig
import tempfile
import threading
import time
from pathlib import Path

__all__ = ["NativeBuildError", "build", "launchers", "library", "library_path", "source_files"]

_SOURCE_DIR = Path(__file__).resolve().parent / "csrc"
_LIBRARY_NAME = "liblalamo_b200_kernels.so"
_NVCC_FLAGS = [
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-O3",
    "-std=c++17",
    "-lineinfo",
    "--shared",
    "-Xcompiler",
    "-fPIC",
    "--expt-relaxed-constexpr",
]

_lock = threading.Lock()
_library: ctypes.CDLL | None = None
_launchers: object | None = None


class NativeBuildError(RuntimeError):
    pass


def source_files() -> list[Path]:
    return sorted(_SOURCE_DIR.glob("*.cu"))


def _source_digest() -> str:
    digest = hashlib.sha256()
    for path in sorted(_SOURCE_DIR.glob("*.cu*")):
        digest.update(path.name.encode())
        digest.update(path.read_bytes())
    digest.update(" ".join(_NVCC_FLAGS).encode())
    digest.update(_wrappers_source().encode())
    return digest.hexdigest()[:16]


def _prototypes() -> dict[str, tuple[str, list[str]]]:
    """The launchers' prototypes as the sources define them: name -> (result type, type of every parameter), all pointers being ``void*``."""
    found: dict[str, tuple[str, list[str]]] = {}
    for path in source_files():
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for result, name, parameters in re.findall(r"^(int|long long) (lb_\w+)\(([^)]*)\)\s*\{", text, re.MULTILINE):
            declared = filter(None, (" ".join(part.split()) for part in parameters.split(",")))
            found[name] = (result, ["void*" if "*" in part or "cudaStream_t" in part else part.rsplit(" ", 1)[0] for part in declared])
    return found


_WRAPPERS_HEAD = """// Made from the launchers' prototypes: a function of the same name and arguments for each, callable from Python.  A pointer is
// None, an address, or anything with a data_ptr() (a tensor); numbers are what ctypes takes for them (wider integers lose their upper
// bits), or ctypes' own objects.
#define Py_LIMITED_API 0x030A0000
#define PY_SSIZE_T_CLEAN
#include <Python.h>

static bool take_integer(PyObject* object, long long* value) {
    PyObject* number = nullptr;
    if (!PyLong_Check(object)) {
        PyObject* held = PyIndex_Check(object) ? nullptr : PyObject_GetAttrString(object, "value");   // a ctypes object's
        if (held == nullptr) PyErr_Clear();
        number = PyNumber_Index(held != nullptr ? held : object);
        Py_XDECREF(held);
        if (number == nullptr) return false;
    }
    *value = static_cast<long long>(PyLong_AsUnsignedLongLongMask(number != nullptr ? number : object));
    Py_XDECREF(number);
    return !(*value == -1 && PyErr_Occurred());
}

static bool take_pointer(PyObject* object, void** value) {
    static PyObject* method = PyUnicode_InternFromString("data_ptr");
    long long address = 0;
    if (object != Py_None) {
        PyObject* held = nullptr;
        if (!PyLong_Check(object)) {
            held = PyObject_HasAttr(object, method) ? PyObject_CallMethodObjArgs(object, method, nullptr) : PyIndex_Check(object) ? PyNumber_Index(object) : PyObject_GetAttrString(object, "value");
            if (held == nullptr) return false;
        }
        const bool taken = held == Py_None || take_integer(held != nullptr ? held : object, &address);   // (None: a null pointer of ctypes)
        Py_XDECREF(held);
        if (!taken) return false;
    }
    *value = reinterpret_cast<void*>(address);
    return true;
}

static bool take_float(PyObject* object, double* value) {
    *value = PyFloat_AsDouble(object);
    if (*value == -1.0 && PyErr_Occurred()) {
        if (!PyErr_ExceptionMatches(PyExc_TypeError)) return false;
        PyObject *type, *error, *trace;
        PyErr_Fetch(&type, &error, &trace);
        PyObject* held = PyObject_GetAttrString(object, "value");   // a ctypes object's
        if (held == nullptr) {
            PyErr_Clear();
            PyErr_Restore(type, error, trace);
            return false;
        }
        Py_XDECREF(type), Py_XDECREF(error), Py_XDECREF(trace);
        *value = PyFloat_AsDouble(held);
        Py_DECREF(held);
    }
    return !(*value == -1.0 && PyErr_Occurred());
}
"""


def _wrappers_source() -> str:
    """C++ source of the wrappers through which Python calls the launchers (a module named ``lalamo_b200_launchers``)."""
    taken_as = {"void*": ("pointer", "void*"), "float": ("float", "double")}
    parts, table = [_WRAPPERS_HEAD], []
    for name, (result, types) in _prototypes().items():
        lines = [f"extern \"C\" {result} {name}({', '.join(types)});",
                 f"static PyObject* wrap_{name}(PyObject*, PyObject* const* arguments, Py_ssize_t count) {{",
                 f"    if (count != {len(types)}) return PyErr_Format(PyExc_TypeError, \"{name} takes {len(types)} arguments, got %zd\", count);"]
        for index, declared in enumerate(types):
            kind, variable = taken_as.get(declared, ("integer", "long long"))
            lines.append(f"    {variable} a{index};\n    if (!take_{kind}(arguments[{index}], &a{index})) return nullptr;")
        call = ", ".join(f"static_cast<{declared}>(a{index})" for index, declared in enumerate(types))
        lines += [f"    {result} code;", "    Py_BEGIN_ALLOW_THREADS", f"    code = {name}({call});", "    Py_END_ALLOW_THREADS", "    return PyLong_FromLongLong(code);", "}"]
        parts.append("\n".join(lines))
        table.append(f"    {{\"{name}\", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(wrap_{name})), METH_FASTCALL, nullptr}},")
    parts.append("static PyMethodDef methods[] = {\n" + "\n".join(table) + "\n    {nullptr, nullptr, 0, nullptr}};\n"
                 'static PyModuleDef module = {PyModuleDef_HEAD_INIT, "lalamo_b200_launchers", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};\n'
                 "PyMODINIT_FUNC PyInit_lalamo_b200_launchers() { return PyModule_Create(&module); }\n")
    return "\n\n".join(parts)


class _CtypesLaunchers:
    """The same through ``ctypes``, for a library built where Python's headers were missing."""

    def __init__(self, loaded: ctypes.CDLL) -> None:
        c_types = {"void*": ctypes.c_void_p, "float": ctypes.c_float, "int": ctypes.c_int, "unsigned": ctypes.c_uint, "long long": ctypes.c_longlong}
        for name, (result, types) in _prototypes().items():
            function = getattr(loaded, name)
            function.restype, function.argtypes = c_types[result], [c_types[declared] for declared in types]
            setattr(self, name, self._taking_tensors(function))

    @staticmethod
    def _taking_tensors(function):
        types = function.argtypes

        def taken(argument, declared):
            if declared is ctypes.c_void_p and hasattr(argument, "data_ptr"):
                return argument.data_ptr()
            return declared(argument.value if isinstance(argument, ctypes._SimpleCData) else argument)

        def call(*arguments):
            if len(arguments) != len(types):
                raise TypeError(f"{function.__name__} takes {len(types)} arguments, got {len(arguments)}")
            return function(*map(taken, arguments, types))

        return call


def _find_nvcc() -> str:
    candidates = [
        os.environ.get("LALAMO_B200_NVCC"),
        shutil.which("nvcc"),
        os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc"),
        "/usr/local/cuda/bin/nvcc",
    ]
    for candidate in candidates:
        if candidate and os.path.isfile(candidate) and os.access(candidate, os.X_OK):
            return candidate
    raise NativeBuildError("nvcc was not found (looked at $LALAMO_B200_NVCC, PATH, $CUDA_HOME/bin, /usr/local/cuda/bin)")


def _build_dirs() -> list[Path]:
    dirs = [Path(__file__).resolve().parent / "_native"]
    user = os.getuid() if hasattr(os, "getuid") else 0
    dirs.append(Path(tempfile.gettempdir()) / f"lalamo_b200_native_{user}")
    return dirs


def _usable(directory: Path) -> bool:
    try:
        directory.mkdir(parents=True, exist_ok=True)
        probe = directory / f".probe_{os.getpid()}"
        probe.write_bytes(b"")
        probe.unlink()
        return True
    except OSError:
        return False


def library_path() -> Path | None:
    """The up-to-date built library, if there is one."""
    digest = _source_digest()
    for directory in _build_dirs():
        candidate = directory / _LIBRARY_NAME
        stamp = directory / "source.digest"
        if candidate.is_file() and stamp.is_file() and stamp.read_text().strip() == digest:
            return candidate
    return None


def build(verbose: bool = True, force: bool = False) -> Path:
    """Compiles every kernel for sm_100a; returns the library's path."""
    existing = None if force else library_path()
    if existing is not None:
        return existing
    nvcc = _find_nvcc()
    directory = next((d for d in _build_dirs() if _usable(d)), None)
    if directory is None:
        raise NativeBuildError(f"none of {[str(d) for d in _build_dirs()]} can be written")
    sources = source_files()
    objects: list[Path] = []
    started = time.time()
    processes: list[tuple[Path, subprocess.Popen]] = []
    compile_flags = [flag for flag in _NVCC_FLAGS if flag != "--shared"]
    wrappers = None
    headers = sysconfig.get_paths()["include"]
    if os.path.isfile(os.path.join(headers, "Python.h")):
        wrappers = directory / f"launchers.{os.getpid()}.cpp"
        wrappers.write_text(_wrappers_source())
        sources = [*sources, wrappers]
        compile_flags += ["-I", headers]
    for source in sources:
        target = directory / (source.stem + f".{os.getpid()}.o")
        objects.append(target)
        command = [nvcc, *compile_flags, "-c", str(source), "-o", str(target)]
        processes.append((source, subprocess.Popen(command, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    if verbose:
        print(f"[lalamo_b200] compiling {len(sources)} CUDA sources for sm_100a into {directory} ...", file=sys.stderr, flush=True)
    for source, process in processes:
        while True:
            try:
                output, _ = process.communicate(timeout=20)
                break
            except subprocess.TimeoutExpired:
                if verbose:
                    print(f"[lalamo_b200] still compiling ({source.name}, {time.time() - started:.0f} s) ...", file=sys.stderr, flush=True)
        if process.returncode != 0:
            for _, other in processes:
                if other.poll() is None:
                    other.kill()
            raise NativeBuildError(f"nvcc failed on {source.name}:\n{output}")
    temporary = directory / f"{_LIBRARY_NAME}.{os.getpid()}.tmp"
    link = subprocess.run(
        [nvcc, "--shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(temporary), *map(str, objects)],
        stdout=subprocess.PIPE,
        stderr=subprocess.STDOUT,
        text=True,
    )
    for target in objects + ([wrappers] if wrappers is not None else []):
        target.unlink(missing_ok=True)
    if link.returncode != 0:
        raise NativeBuildError(f"linking the kernel library failed:\n{link.stdout}")
    os.replace(temporary, directory / _LIBRARY_NAME)
    (directory / "source.digest").write_text(_source_digest())
    if verbose:
        print(f"[lalamo_b200] built {_LIBRARY_NAME} in {time.time() - started:.0f} s", file=sys.stderr, flush=True)
    return directory / _LIBRARY_NAME


def library() -> ctypes.CDLL:
    """The loaded kernel library (built at the first call if needed)."""
    global _library
    with _lock:
        if _library is None:
            path = build()
            try:
                _library = ctypes.CDLL(str(path))
            except OSError as error:
                raise NativeBuildError(f"cannot load {path}: {error}") from error
        return _library


def launchers() -> object:
    """The library's launchers as functions: a pointer may be given as a tensor, ``None`` or an address, numbers as they are."""
    global _launchers
    loaded = library()
    with _lock:
        if _launchers is None:
            if hasattr(loaded, "PyInit_lalamo_b200_launchers"):
                loader = importlib.machinery.ExtensionFileLoader("lalamo_b200_launchers", loaded._name)
                _launchers = importlib.util.module_from_spec(importlib.util.spec_from_loader("lalamo_b200_launchers", loader))
                loader.exec_module(_launchers)
            else:
                _launchers = _CtypesLaunchers(loaded)
        return _launchers
