"""In-tree build of the sm_100a CUDA library (``libflashrt_b200.so``) with nvcc.

The library is a plain C-ABI shared object: no torch, no pybind.  nvcc
cross-compiles for sm_100a without a GPU, so this also runs on a CPU-only box.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libflashrt_b200.so")
CALLS = os.path.join(HERE, "_native_calls" + sysconfig.get_config_var("EXT_SUFFIX"))     # one per interpreter version
OBJ = os.path.join(CSRC, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def sources() -> list[str]:
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def calls_source(protos: dict[str, list[str]]) -> str:
    """C source of the extension module that calls the entry points: one function per prototype, positional arguments.

    A small product is bound by the host: through ctypes a call with 14-16 arguments costs 2.5-3 us on top of its launch
    (attribute lookup, one converter object per argument), the vectorcall functions written here about 0.3 us.  A pointer is
    an int or None, a number an int or a float; anything else (a ctypes object, a wrong count) returns NotImplemented and the
    caller takes the ctypes path, which converts or refuses it as it always did.  The GIL is released around the call."""
    cnum = {"int": ("long long", "PyLong_Check", "PyLong_AsLongLong"),
            "long long": ("long long", "PyLong_Check", "PyLong_AsLongLong"),
            "unsigned": ("long long", "PyLong_Check", "PyLong_AsLongLong"),
            "unsigned long long": ("unsigned long long", "PyLong_Check", "PyLong_AsUnsignedLongLong"),
            "ptr": ("unsigned long long", "PyLong_Check", "PyLong_AsUnsignedLongLong"),
            "float": ("double", "PyFloat_Check", "PyFloat_AsDouble")}
    out = ["#define PY_SSIZE_T_CLEAN", "#include <Python.h>", ""]
    table = []
    for name, types in protos.items():
        n = len(types)
        ctypes_ = ["const void*" if t == "ptr" else t for t in types]
        out.append(f"int {name}({', '.join(ctypes_) or 'void'});")
        out.append(f"static PyObject* w_{name}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{")
        out.append(f"    if (n != {n}) Py_RETURN_NOTIMPLEMENTED;")
        for i, t in enumerate(types):
            c, check, conv = cnum[t]
            out.append(f"    {c} v{i} = 0;")
            if t == "ptr":
                out.append(f"    if (a[{i}] != Py_None) {{ if (!{check}(a[{i}])) Py_RETURN_NOTIMPLEMENTED; "
                           f"v{i} = {conv}(a[{i}]); }}")
            elif t == "float":
                out.append(f"    if (PyFloat_Check(a[{i}])) v{i} = PyFloat_AS_DOUBLE(a[{i}]); "
                           f"else if (PyLong_Check(a[{i}])) v{i} = PyLong_AsDouble(a[{i}]); else Py_RETURN_NOTIMPLEMENTED;")
            else:
                out.append(f"    if (!{check}(a[{i}])) Py_RETURN_NOTIMPLEMENTED; v{i} = {conv}(a[{i}]);")
        if n:
            out.append("    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NOTIMPLEMENTED; }")
        args = ", ".join(f"(const void*)(uintptr_t)v{i}" if t == "ptr" else f"({t})v{i}" for i, t in enumerate(types))
        out.append("    int rc;")
        out.append(f"    Py_BEGIN_ALLOW_THREADS rc = {name}({args}); Py_END_ALLOW_THREADS")
        out.append("    return PyLong_FromLong(rc);\n}")
        table.append(f'    {{"{name}", (PyCFunction)(void*)w_{name}, METH_FASTCALL, NULL}},')
    out += ["static PyMethodDef methods[] = {", *table, "    {NULL, NULL, 0, NULL}};",
            'static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native_calls", NULL, -1, methods};',
            "PyMODINIT_FUNC PyInit__native_calls(void) { return PyModule_Create(&module); }", ""]
    return "\n".join(out)


def build_calls(force: bool = False) -> str | None:
    """The extension module behind ``_lib.call``; None where the interpreter's headers or a C compiler are missing (the ctypes
    path then serves every call).  A module of another header or library, or one without an interpreter tag (any version
    would import it), does not stay behind."""
    from ._lib import HEADER_PATH, parse_header
    inc, cc = sysconfig.get_paths()["include"], shutil.which("gcc") or shutil.which("cc")
    stale = force or _stale(CALLS, [HEADER_PATH, os.path.abspath(__file__), LIB])
    untagged = os.path.join(os.path.dirname(CALLS), "_native_calls.so")
    for old in {untagged, CALLS} if stale else {untagged} - {CALLS}:
        if os.path.exists(old):
            os.remove(old)
    if cc is None or not os.path.exists(os.path.join(inc, "Python.h")):
        return None if stale else CALLS
    if stale:
        src = os.path.join(OBJ, "native_calls.c")
        with open(src, "w") as f:
            f.write(calls_source(parse_header()))
        r = subprocess.run([cc, "-O2", "-fPIC", "-shared", "-I", inc, src, "-o", CALLS, "-L", HERE, "-l:libflashrt_b200.so",
                            "-Wl,-rpath,$ORIGIN"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("gcc failed:\n" + r.stdout + r.stderr)
    return CALLS


def _nvcc() -> str:
    n = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(n):
        raise RuntimeError("nvcc not found; the sm_100a library cannot be built")
    return n


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build_native(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` and link ``libflashrt_b200.so``.  Returns its path.

    ``FRT_NVCC_EXTRA`` (environment, space separated) appends compiler flags, e.g. ``-DFRT_PHASE_STAMPS`` for the
    device-timer phase stamps that ``bench.py --workload timeline`` reads through ``frt_b200_phase_stamps_read`` (use
    ``--force`` when switching it on or off: the objects do not depend on the environment)."""
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    extra = os.environ.get("FRT_NVCC_EXTRA", "").split()
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(os.path.dirname(HERE), "include", "flashrt_b200.h"))
    headers = [h for h in headers if os.path.exists(h)]
    jobs = []
    objs = []
    for s in sources():
        src = os.path.join(CSRC, s)
        obj = os.path.join(OBJ, s[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc] + NVCC_FLAGS + extra + ["-I", os.path.join(os.path.dirname(HERE), "include"), "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            logs = list(ex.map(run, jobs))
        if verbose:
            print("\n".join(logs))
    if jobs or force or _stale(LIB, objs):
        run([nvcc, "-shared", "-o", LIB] + objs)
    build_calls(force)
    return LIB


if __name__ == "__main__":
    import sys
    print(build_native(force="--force" in sys.argv, verbose="-v" in sys.argv))
