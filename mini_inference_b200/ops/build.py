"""Builds the CUDA sources under csrc/ into one shared library next to the package, for
sm_100a only, with nvcc directly (no JIT cache outside the tree, nothing needed from the
network or from HOME).  The library is rebuilt when a source changed; otherwise it is loaded
as it lies.  The first call of a fresh checkout compiles, printing a line per source file.

Beside it lies a Python extension with a function per C entry point (host_calls), generated from
their declarations: the engine calls the library through it.  A call with 25 arguments, twelve of
them tensors, costs the host 4.0 us through ctypes and 1.0 us that way, and a mixer of a few
hundred tokens waits for the host.  Where it cannot be built (no Python headers, no C compiler) the
same calls go through ctypes."""
from __future__ import annotations

import contextlib
import hashlib
import json
import os
import re
import shutil
import subprocess
import sys
import sysconfig
import time
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(PKG, "csrc")


def _out_dir() -> str:
    """The package folder; a per-user folder under the temporary directory when the checkout
    is read-only for this user."""
    if os.access(PKG, os.W_OK):
        return PKG
    import tempfile
    d = os.path.join(tempfile.gettempdir(), f"mini_inference_b200_build_{os.getuid()}")
    os.makedirs(d, exist_ok=True)
    return d


BUILD = os.path.join(_out_dir(), "_build")
LIB = os.path.join(_out_dir(), "_kernels.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr"]
NVCC_FLAGS += os.environ.get("MI_NVCC_EXTRA", "").split()        # e.g. -DMI_ATT_TIMING for the kernels' phase counters


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.isfile(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA kernels of mini_inference_b200 cannot be built")


HOST_CALLS = os.path.join(_out_dir(), "_host_calls" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
POINTER, INTEGER, REAL = "pointer", "integer", "real"


def signatures():
    """{name: (C return type, [(C type, kind of argument)])} of the library's entry points, as csrc/ declares them."""
    out = {}
    for src in _sources():
        with open(os.path.join(CSRC, src)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for ret, name, args in re.findall(r"MI_EXPORT\s+(int|long long)\s+(mi_\w+)\s*\(([^)]*)\)", text):
            kinds = []
            for a in (" ".join(x.split()) for x in args.split(",") if x.strip()):
                ctype = re.sub(r"\s*\w+$", "", a) if not a.endswith("*") else a
                if "*" in ctype or ctype == "cudaStream_t":
                    kinds.append(("void*", POINTER))
                elif ctype in ("int", "long long"):
                    kinds.append((ctype, INTEGER))
                elif ctype == "float":
                    kinds.append((ctype, REAL))
                else:
                    raise RuntimeError(f"{src}: argument type '{ctype}' of {name} has no conversion")
            out[name] = (ret, kinds)
    return out


_HOST_SOURCE = """#include <Python.h>
static PyObject* s_data_ptr;
/* a tensor, an address, an object with a `value` (what ctypes wraps numbers in) or None */
static void* as_pointer(PyObject* o) {
    PyObject* r;
    void* p;
    if (o == Py_None) return NULL;
    if (PyLong_Check(o)) return PyLong_AsVoidPtr(o);
    r = PyObject_CallMethodNoArgs(o, s_data_ptr);
    if (!r && PyErr_ExceptionMatches(PyExc_AttributeError)) {
        PyErr_Clear();
        r = PyObject_GetAttrString(o, "value");
    }
    if (!r) return NULL;
    p = r == Py_None ? NULL : PyLong_AsVoidPtr(r);
    Py_DECREF(r);
    return p;
}
static PyObject* number(PyObject* o) {
    if (PyLong_Check(o) || PyFloat_Check(o) || PyIndex_Check(o) || PyNumber_Check(o)) { Py_INCREF(o); return o; }
    return PyObject_GetAttrString(o, "value");
}
static long long as_integer(PyObject* o) {
    long long v;
    if (PyLong_Check(o)) return PyLong_AsLongLong(o);
    o = number(o);
    if (!o) return -1;
    if (PyFloat_Check(o)) { PyErr_SetString(PyExc_TypeError, "an integer is required"); v = -1; } else v = PyLong_AsLongLong(o);
    Py_DECREF(o);
    return v;
}
static double as_real(PyObject* o) {
    double v;
    if (PyFloat_Check(o)) return PyFloat_AS_DOUBLE(o);
    o = number(o);
    if (!o) return -1.0;
    v = PyFloat_AsDouble(o);
    Py_DECREF(o);
    return v;
}
static int wrong_count(const char* name, Py_ssize_t got, int want) {
    if (got == want) return 0;
    PyErr_Format(PyExc_TypeError, "%s takes %d arguments (%zd given)", name, want, got);
    return 1;
}
"""


def _host_source() -> str:
    """The extension's C source: a typed function per entry point, and bind(name, address)."""
    out, table = [_HOST_SOURCE], []
    take = {POINTER: "as_pointer(v[%d])", INTEGER: "(%s)as_integer(v[%d])", REAL: "(float)as_real(v[%d])"}
    for name, (ret, args) in signatures().items():
        types = ", ".join(t for t, _ in args) or "void"
        lines = [f"static {ret} (*p_{name})({types});",
                 f"static PyObject* w_{name}(PyObject* self, PyObject* const* v, Py_ssize_t n) {{", f"    {ret} r;"]
        lines += [f"    {t} a{i};" for i, (t, _) in enumerate(args)]
        lines.append(f'    if (wrong_count("{name}", n, {len(args)})) return NULL;')
        for i, (t, kind) in enumerate(args):
            lines.append(f"    a{i} = " + (take[kind] % ((t, i) if kind == INTEGER else i)) + f"; if ({'!' if kind == POINTER else '-1 == '}a{i} && PyErr_Occurred()) return NULL;")
        lines += ["    Py_BEGIN_ALLOW_THREADS", f"    r = p_{name}({', '.join(f'a{i}' for i in range(len(args)))});",
                  "    Py_END_ALLOW_THREADS", "    return PyLong_FromLongLong(r);", "}"]
        out.append("\n".join(lines))
        table.append(name)
    out.append("static PyObject* bind(PyObject* self, PyObject* const* v, Py_ssize_t n) {\n    const char* name;\n    void* at;\n"
               '    if (wrong_count("bind", n, 2) || !(name = PyUnicode_AsUTF8(v[0])) || !(at = as_pointer(v[1]))) return NULL;')
    out += [f'    if (!strcmp(name, "{n}")) {{ *(void**)&p_{n} = at; Py_RETURN_NONE; }}' for n in table]
    out.append("    PyErr_SetString(PyExc_KeyError, name);\n    return NULL;\n}\nstatic PyMethodDef methods[] = {\n"
               '    {"bind", (PyCFunction)(void*)bind, METH_FASTCALL, NULL},')
    out += [f'    {{"{n}", (PyCFunction)(void*)w_{n}, METH_FASTCALL, NULL}},' for n in table]
    out.append("    {NULL, NULL, 0, NULL}};\nstatic struct PyModuleDef module = {PyModuleDef_HEAD_INIT, \"_host_calls\", NULL, -1, methods};\n"
               'PyMODINIT_FUNC PyInit__host_calls(void) {\n    s_data_ptr = PyUnicode_InternFromString("data_ptr");\n    return PyModule_Create(&module);\n}\n')
    return "\n".join(out)


def _build_host_calls() -> None:
    cc = next((c for c in (os.environ.get("CC"), "cc", "gcc", "clang") if c and shutil.which(c)), None)
    include = sysconfig.get_paths()["include"]
    with contextlib.suppress(FileNotFoundError):
        os.remove(HOST_CALLS)                                   # never an older one beside a new library
    if cc is None or not os.path.isfile(os.path.join(include, "Python.h")):
        _log("no C compiler or no Python headers: the entry points are called through ctypes")
        return
    tmp = HOST_CALLS + f".tmp{os.getpid()}"
    r = subprocess.run([cc, "-O2", "-shared", "-fPIC", "-I", include, "-x", "c", "-", "-o", tmp], input=_host_source(), capture_output=True, text=True)
    if r.returncode != 0:
        _log(f"{cc} failed on host_calls.c, the entry points are called through ctypes:\n{r.stderr[-2000:]}")
        return
    os.replace(tmp, HOST_CALLS)


def host_calls():
    """The extension of the library that lies beside it, or None."""
    if not os.path.isfile(HOST_CALLS):
        return None
    import importlib.util
    spec = importlib.util.spec_from_file_location("_host_calls", HOST_CALLS)
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _digest() -> str:
    h = hashlib.sha256((" ".join(NVCC_FLAGS) + os.path.basename(HOST_CALLS) + _host_source()).encode())
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(CSRC, f), "rb") as fh:
                h.update(f.encode() + b"\0" + fh.read())
    return h.hexdigest()


def _log(msg):
    print(f"[mini_inference_b200 build] {msg}", file=sys.stderr, flush=True)


def is_current() -> bool:
    stamp = os.path.join(BUILD, "stamp.json")
    if not (os.path.isfile(LIB) and os.path.isfile(stamp)):
        return False
    try:
        with open(stamp) as f:
            return json.load(f).get("digest") == _digest()
    except (OSError, ValueError):
        return False


def build(force: bool = False, verbose: bool = True) -> str:
    """Compile every .cu under csrc/ (in parallel) and link _kernels.so.  Returns its path."""
    if not force and is_current():
        if not os.path.isfile(HOST_CALLS):                      # a library that came without it
            _build_host_calls()
        return LIB
    nvcc = _nvcc()
    os.makedirs(BUILD, exist_ok=True)
    sources = _sources()
    t0 = time.time()
    if verbose:
        _log(f"compiling {len(sources)} CUDA sources for sm_100a with {nvcc} (first call only)")

    def compile_one(src):
        obj = os.path.join(BUILD, src[:-3] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            _log(f"  compiled {src} ({time.time() - t0:.0f}s)")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as pool:
        objs = list(pool.map(compile_one, sources))
    tmp = LIB + f".tmp{os.getpid()}"
    r = subprocess.run([nvcc, "-shared", "-o", tmp, *objs, "-lcudart"], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"linking _kernels.so failed:\n{r.stdout}\n{r.stderr}")
    os.replace(tmp, LIB)
    _build_host_calls()
    with open(os.path.join(BUILD, "stamp.json"), "w") as f:
        json.dump({"digest": _digest(), "sources": sources}, f)
    if verbose:
        _log(f"built {LIB} in {time.time() - t0:.0f}s")
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv)
