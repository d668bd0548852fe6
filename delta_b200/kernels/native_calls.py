"""The library's launchers as functions of a CPython module, for the host's time in steps that are not replayed.

A launcher takes up to thirty numbers and addresses, which ``ctypes`` turns over one by one: 3.8 us for 22 of them, half of what a small launch
costs the host.  From the signatures a C file is written that does the same with the interpreter's own calls (0.2 us), and compiled beside the
library.  It holds no kernel: it calls the library's functions by address, without the interpreter's lock as ``ctypes`` does.  Where it cannot be
compiled or loaded, a warning says why and the launchers are called through ``ctypes``.
"""
from __future__ import annotations

import ctypes as C
import hashlib
import importlib.machinery
import importlib.util
import os
import shlex
import shutil
import subprocess
import sysconfig
import warnings
from pathlib import Path
from typing import Dict, Optional

# argument type -> (C type, conversion of ``a[i]``)
_TYPES = {C.c_void_p: ("void*", "address"), C.c_int: ("int", "whole"), C.c_longlong: ("long long", "whole"), C.c_float: ("float", "real"),
          C.c_double: ("double", "real")}

_HEAD = r"""
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>

// Integers wrap to the width of their argument, as ctypes has them; numbers of other types give their index or float value.
static unsigned long long whole(PyObject* o) {
  if (PyLong_Check(o)) return PyLong_AsUnsignedLongLongMask(o);
  PyObject* i = PyNumber_Index(o);
  if (i == NULL) return 0;
  unsigned long long v = PyLong_AsUnsignedLongLongMask(i);
  Py_DECREF(i);
  return v;
}
static void* address(PyObject* o) { return o == Py_None ? NULL : (void*)(uintptr_t)whole(o); }
static double real(PyObject* o) { return PyFloat_AsDouble(o); }
static int wrong_count(const char* name, Py_ssize_t got, int want) {
  if (got == want) return 0;
  PyErr_Format(PyExc_TypeError, "%s takes %d arguments, not %zd", name, want, got);
  return 1;
}
"""


def _source(signatures: Dict[str, list]) -> str:
    out, table, look = [_HEAD], [], []
    for name, args in signatures.items():
        types = [_TYPES[a][0] for a in args]
        out.append(f"static int (*p_{name})({', '.join(types) or 'void'});")
        out.append(f"static PyObject* f_{name}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{")
        out.append(f'  (void)self; (void)a;\n  if (wrong_count("{name}", n, {len(args)})) return NULL;')
        out += [f"  {t} v{i} = ({t}){_TYPES[args[i]][1]}(a[{i}]);" for i, t in enumerate(types)]
        out.append("  if (PyErr_Occurred()) return NULL;\n  int r;\n  Py_BEGIN_ALLOW_THREADS")
        out.append(f"  r = p_{name}({', '.join(f'v{i}' for i in range(len(args)))});")
        out.append("  Py_END_ALLOW_THREADS\n  return PyLong_FromLong(r);\n}")
        table.append(f'  {{"{name}", (PyCFunction)(void (*)(void))f_{name}, METH_FASTCALL, NULL}},')
        look.append(f'  if ((*(void**)&p_{name} = dlsym(h, "{name}")) == NULL) {{ PyErr_SetString(PyExc_ImportError, "no {name} in the library"); return NULL; }}')
    out.append("static PyObject* connect(PyObject* self, PyObject* arg) {\n  (void)self;\n  void* h = PyLong_AsVoidPtr(arg);\n  if (PyErr_Occurred()) return NULL;")
    out += look + ["  Py_RETURN_NONE;\n}"]
    out.append("static PyMethodDef methods[] = {\n" + "\n".join(table) + '\n  {"connect", connect, METH_O, NULL},\n  {NULL, NULL, 0, NULL}\n};')
    out.append('static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "dk_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};')
    out.append("PyMODINIT_FUNC PyInit_dk_calls(void) { return PyModule_Create(&module); }")
    return "\n".join(out) + "\n"


def _compile(source: str, to: Path) -> str:
    """An empty text, or why there is no module."""
    include = sysconfig.get_paths()["include"]
    cc = shlex.split(os.environ.get("CC") or "") or [c for c in (shutil.which("gcc"), shutil.which("cc")) if c][:1]      # (CC may bring arguments)
    if not cc:
        return "there is no C compiler"
    if not (Path(include) / "Python.h").is_file():
        return f"there is no Python.h in {include}"
    c, tmp = to.with_suffix(f".{os.getpid()}.c"), to.with_suffix(f".{os.getpid()}.tmp")
    try:
        c.write_text(source)
        r = subprocess.run([*cc, "-O2", "-shared", "-fPIC", "-I", include, str(c), "-o", str(tmp), "-ldl"], capture_output=True, text=True)
        if r.returncode != 0:
            return f"{shlex.join(cc)} ended with {r.returncode}: {r.stderr.strip()[-500:]}"
        os.replace(tmp, to)
        return ""
    except OSError as e:
        return str(e)
    finally:
        c.unlink(missing_ok=True)
        tmp.unlink(missing_ok=True)


def load(library: C.CDLL, path: Path, signatures: Dict[str, list]) -> Optional[dict]:
    """{launcher: function} for those of ``signatures`` that take numbers and addresses only; None, with a warning, where there is no module."""
    plain = {name: args for name, args in signatures.items() if all(a in _TYPES for a in args)}
    source = _source(plain)
    so = Path(path).parent / ("dk_calls_" + hashlib.sha256((source + sysconfig.get_config_var("EXT_SUFFIX")).encode()).hexdigest()[:16]
                              + sysconfig.get_config_var("EXT_SUFFIX"))
    why = "" if so.is_file() else _compile(source, so)
    if not why:
        try:
            loader = importlib.machinery.ExtensionFileLoader("dk_calls", str(so))
            module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("dk_calls", str(so), loader=loader))
            loader.exec_module(module)
            module.connect(library._handle)
            return {name: getattr(module, name) for name in plain}
        except ImportError as e:
            why = str(e)
    warnings.warn(f"the launchers are called through ctypes, which costs the host about 4 us a launch: {why}", RuntimeWarning, stacklevel=2)
    return None
