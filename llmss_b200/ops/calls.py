"""Entries of the kernel library as plain Python functions: an extension module written from their signatures.

A ctypes call converts every argument through an object of its own: 3.2 us for the 24 arguments of a linear layer, of which a decode step issues hundreds;
through the module it is 0.4 us.  What the module does not take (a ctypes object, a wrong number or kind of arguments) it hands to the ctypes function, which
behaves and raises as before; without the module (no compiler, no Python headers, a folder that takes no files) every call goes there.
"""
from __future__ import annotations

import ctypes as C
import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

NAME = "_llmss_calls"
_TYPES = {C.c_void_p: "void*", C.c_int: "int", C.c_int64: "int64_t", C.c_float: "float", C.c_size_t: "size_t"}
_RESULTS = {C.c_int: "PyLong_FromLong", C.c_int64: "PyLong_FromLongLong"}

_HEAD = """// generated from the signatures of the library's entries
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

// argument i as a C value; 0: not a plain number (the ctypes function decides)
static int get_ptr(PyObject* o, void** v) {
  if (o == Py_None) { *v = 0; return 1; }
  if (!PyLong_Check(o)) return 0;
  *v = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(o);
  return !PyErr_Occurred();
}
static int get_int(PyObject* o, uint64_t* v) {
  if (!PyLong_Check(o)) return 0;
  *v = PyLong_AsUnsignedLongLongMask(o);
  return !PyErr_Occurred();
}
static int get_float(PyObject* o, float* v) {
  if (!PyFloat_Check(o)) return 0;
  *v = (float)PyFloat_AS_DOUBLE(o);
  return 1;
}
static PyObject* otherwise(PyObject* f, PyObject* const* a, Py_ssize_t n) {
  PyErr_Clear();
  if (!f) { PyErr_SetString(PyExc_RuntimeError, "entry is not bound"); return 0; }
  return PyObject_Vectorcall(f, a, (size_t)n, 0);
}
"""


def wrappable(sigs: dict) -> list:
    """Names whose arguments and result are plain numbers and addresses."""
    return [n for n, (res, args) in sigs.items() if res in _RESULTS and args and all(a in _TYPES for a in args)]


def source(sigs: dict) -> str:
    out, table, binds = [_HEAD], [], []
    for k, name in enumerate(wrappable(sigs)):
        res, args = sigs[name]
        cres = _TYPES[res]
        decl, get, use = [], [], []
        for i, a in enumerate(args):
            if a is C.c_void_p:
                decl.append(f"void* v{i};")
                get.append(f"get_ptr(a[{i}], &v{i})")
                use.append(f"v{i}")
            elif a is C.c_float:
                decl.append(f"float v{i};")
                get.append(f"get_float(a[{i}], &v{i})")
                use.append(f"v{i}")
            else:
                decl.append(f"uint64_t v{i};")
                get.append(f"get_int(a[{i}], &v{i})")
                use.append(f"({_TYPES[a]})v{i}")
        out.append(f"""
static {cres} (*f{k})({", ".join(_TYPES[a] for a in args)});
static PyObject* o{k};
static PyObject* w{k}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{
  {" ".join(decl)}
  if (n != {len(args)} || !f{k} || !({" && ".join(get)})) return otherwise(o{k}, a, n);
  {cres} r;
  Py_BEGIN_ALLOW_THREADS
  r = f{k}({", ".join(use)});
  Py_END_ALLOW_THREADS
  return {_RESULTS[res]}(r);
}}""")
        table.append(f'  {{"{name}", (PyCFunction)(void*)w{k}, METH_FASTCALL, 0}},')
        binds.append(f"    case {k}: f{k} = address; Py_XSETREF(o{k}, f); break;")
    out.append("""
static PyObject* bind_entry(PyObject* self, PyObject* args) {
  int k; unsigned long long at; PyObject* f;
  if (!PyArg_ParseTuple(args, "iKO", &k, &at, &f)) return 0;
  void* address = (void*)(uintptr_t)at;
  Py_INCREF(f);
  switch (k) {
""" + "\n".join(binds) + """
    default: Py_DECREF(f); PyErr_SetString(PyExc_IndexError, "no such entry"); return 0;
  }
  Py_RETURN_NONE;
}
static PyMethodDef methods[] = {
""" + "\n".join(table) + """
  {"bind", bind_entry, METH_VARARGS, 0},
  {0, 0, 0, 0}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "NAME", 0, -1, methods};
PyMODINIT_FUNC PyInit_NAME(void) { return PyModule_Create(&module); }
""".replace("NAME", NAME))
    return "\n".join(out)


def _abi() -> str:
    return sysconfig.get_config_var("SOABI") or "abi"


def module_path(lib_dir: Path, sigs: dict) -> Path:
    """The file carries its source's digest and Python's ABI: one written from other signatures, or for another Python, is never loaded."""
    return Path(lib_dir) / f"{NAME}.{hashlib.sha256(source(sigs).encode()).hexdigest()[:16]}.{_abi()}.so"


def compiler():
    """(C compiler, folder of Python.h), or None where the module cannot be built."""
    cc, include = shutil.which("gcc") or shutil.which("cc"), sysconfig.get_paths()["include"]
    return (cc, include) if cc is not None and (Path(include) / "Python.h").exists() else None


def build(lib_dir: Path, obj_dir: Path, sigs: dict) -> bool:
    """Compile the module if it is not there; False without a compiler or Python's headers."""
    path = module_path(lib_dir, sigs)
    if path.exists():
        return True
    tools = compiler()
    if tools is None:
        return False
    text, tmp = Path(obj_dir) / f"{NAME}.c", path.with_suffix(f".tmp{os.getpid()}")
    text.write_text(source(sigs))
    r = subprocess.run([tools[0], "-O2", "-shared", "-fPIC", "-I", tools[1], str(text), "-o", str(tmp)], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{tools[0]} failed for {text}:\n{r.stderr}")
    for old in Path(lib_dir).glob(f"{NAME}.*.{_abi()}.so"):       # (another Python's stay)
        old.unlink()
    os.replace(tmp, path)
    return True


def attach(lib, lib_dir: Path, sigs: dict) -> int:
    """Replace the ctypes functions of ``lib`` that the module has; how many."""
    path = module_path(lib_dir, sigs)
    if not path.exists():
        return 0
    try:
        spec = importlib.util.spec_from_loader(NAME, importlib.machinery.ExtensionFileLoader(NAME, str(path)))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
    except ImportError as e:
        print(f"[llmss_b200] library calls go through ctypes: {e}", file=sys.stderr)
        return 0
    names = wrappable(sigs)
    for k, name in enumerate(names):
        if hasattr(lib, name):
            fn = getattr(lib, name)
            mod.bind(k, C.cast(fn, C.c_void_p).value, fn)
            setattr(lib, name, getattr(mod, name))
    return len(names)
