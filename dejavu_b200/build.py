"""Builds the C-ABI libraries of sm_100a kernels in-tree with nvcc.

    python -m dejavu_b200.build [--force] [--verbose] [--lib sparse|hybrid|routed]

  sparse  libdejavu_b200.so         the contextual-sparse OPT decode path
  hybrid  libdejavu_b200_hybrid.so  gated linear attention, sliding-window attention, hyper-connected streams
  routed  libdejavu_b200_routed.so  matrix memories, latent attention, routed feed-forwards

Each .cu file is compiled to an object in parallel, then linked into the shared libraries that sit next to this file. Beside them
stands _calls, a small extension module with a binding for each signature of the libraries' functions (_lib.py): a call with 17
arguments takes 0.5 us through it and 3 us through ctypes, which serves where it could not be compiled.
Nothing is cached outside the package directory. A library can be built alone, so that a program that serves one kind
of model compiles only what it needs.
"""
from __future__ import annotations

import argparse
import os
import shlex
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "build"
LIB = PKG / "libdejavu_b200.so"
HYBRID_LIB = PKG / "libdejavu_b200_hybrid.so"
ROUTED_LIB = PKG / "libdejavu_b200_routed.so"
LIBS = {"sparse": LIB, "hybrid": HYBRID_LIB, "routed": ROUTED_LIB}

# translation units of the hybrid decoders' libraries; those both use are compiled once and linked into both
_BOTH = ("api", "hybrid_gemv", "hybrid_residual", "hybrid_rotary", "hybrid_window_simple", "hybrid_window_prefill")
_UNITS = {"hybrid": _BOTH + ("hybrid_attention", "hybrid_gla", "hybrid_gla_mma"),
          "routed": _BOTH + ("hybrid_mlstm", "hybrid_mlstm_prefill", "hybrid_latent", "hybrid_latent_decode", "hybrid_moe",
                             "hybrid_moe_gemm")}

NVCC_FLAGS = [
    "-O3",
    "-std=c++17",
    "-gencode",
    "arch=compute_100a,code=sm_100a",
    "-lineinfo",
    "-Xcompiler",
    "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC=/path/to/nvcc")


def sources(lib: str | None = None) -> list[Path]:
    """Translation units of a library (of all, without a name). api.cu, the plumbing, is part of each."""
    out = sorted(CSRC.glob("*.cu"))
    if lib is None:
        return out
    if lib in _UNITS:
        return [p for p in out if p.stem in _UNITS[lib]]
    return [p for p in out if not p.stem.startswith("hybrid_")]


CALLS = PKG / ("_calls" + sysconfig.get_config_var("EXT_SUFFIX"))

_C_TYPES = {"i": "int", "p": "void *", "l": "long long", "z": "size_t", "f": "float"}
_C_PRELUDE = """#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <limits.h>
#include <stdint.h>

/* 1: converted; 0: not a number of the kind, or too large for it */
static int whole(PyObject *o, long long lo, long long hi, long long *out) {
  int over = 0;
  if (!PyLong_Check(o)) return 0;
  *out = PyLong_AsLongLongAndOverflow(o, &over);
  return !over && *out >= lo && *out <= hi;
}
static int pointer(PyObject *o, void **out) {
  if (o == Py_None) {
    *out = NULL;
    return 1;
  }
  if (!PyLong_Check(o)) return 0;
  *out = PyLong_AsVoidPtr(o);
  if (*out == NULL && PyErr_Occurred()) {
    PyErr_Clear();
    return 0;
  }
  return 1;
}
static int real(PyObject *o, float *out) {
  double v;
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return 0;
  v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    return 0;
  }
  *out = (float)v;
  return 1;
}
"""
_C_CONVERT = {"i": "if (!whole(a[{k}], INT_MIN, INT_MAX, &n)) goto other;\n  v{k} = (int)n;",
              "l": "if (!whole(a[{k}], LLONG_MIN, LLONG_MAX, &n)) goto other;\n  v{k} = n;",
              "z": "if (!whole(a[{k}], 0, LLONG_MAX, &n)) goto other;\n  v{k} = (size_t)n;",
              "p": "if (!pointer(a[{k}], &v{k})) goto other;", "f": "if (!real(a[{k}], &v{k})) goto other;"}


def _binding_source(kinds) -> str:
    """C source of _calls: a function per signature whose `self` is a capsule with the address, and bind(kind, address). The
    interpreter lock is released around a call, as ctypes does."""
    out = [_C_PRELUDE]
    for number, kind in enumerate(kinds):
        res, args = kind[0], kind[1:]
        names = ", ".join(f"v{k}" for k in range(len(args)))
        out.append(f"static PyObject *call{number}(PyObject *self, PyObject *const *a, Py_ssize_t count) {{")
        out.append(f"  {_C_TYPES[res]} (*fn)({', '.join(_C_TYPES[t] for t in args) or 'void'});")
        out += [f"  {_C_TYPES[t]} v{k};" for k, t in enumerate(args)]
        out.append(f"  {_C_TYPES[res]} r;\n  long long n = 0;\n  (void)n;\n  if (count != {len(args)}) goto other;")
        out += ["  " + _C_CONVERT[t].format(k=k) for k, t in enumerate(args)]
        out.append("  *(void **)&fn = PyCapsule_GetPointer(self, NULL);\n  Py_BEGIN_ALLOW_THREADS")
        out.append(f"  r = fn({names});\n  Py_END_ALLOW_THREADS")
        out.append(f"  return {'PyLong_FromLong(r)' if res == 'i' else 'PyLong_FromSize_t(r)'};")
        out.append("other:\n  Py_RETURN_NOTIMPLEMENTED;\n}")
    out.append("static PyMethodDef calls[] = {")
    out += [f'  {{"{kind}", (PyCFunction)(void (*)(void))call{n}, METH_FASTCALL, NULL}},' for n, kind in enumerate(kinds)]
    out.append("""  {NULL, NULL, 0, NULL}};
static PyObject *bind(PyObject *self, PyObject *args) {
  int kind;
  unsigned long long address;
  PyObject *capsule, *fn;
  (void)self;
  if (!PyArg_ParseTuple(args, "iK", &kind, &address)) return NULL;
  if (kind < 0 || kind >= (int)(sizeof(calls) / sizeof(calls[0])) - 1 || address == 0) {
    PyErr_SetString(PyExc_ValueError, "bind: no such kind, or no address");
    return NULL;
  }
  capsule = PyCapsule_New((void *)(uintptr_t)address, NULL, NULL);
  if (capsule == NULL) return NULL;
  fn = PyCFunction_NewEx(&calls[kind], capsule, NULL);
  Py_DECREF(capsule);
  return fn;
}
static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "bind(kind, address): the function there"}, {NULL, NULL, 0, NULL}};
static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", NULL, -1, methods, NULL, NULL, NULL, NULL};
PyMODINIT_FUNC PyInit__calls(void) {
  PyObject *m = PyModule_Create(&module);
  if (m != NULL && PyModule_AddStringConstant(m, "KINDS", KINDS) < 0) {
    Py_DECREF(m);
    return NULL;
  }
  return m;
}
""".replace('"KINDS", KINDS', '"KINDS", "' + " ".join(kinds) + '"'))
    return "\n".join(out)


def build_calls(force: bool = False) -> Path | None:
    """Generates and compiles _calls, the bindings of the libraries' functions. Where that cannot be done (no C compiler, no
    headers of the interpreter) the calls go through ctypes: said, and no error."""
    from . import _lib

    if not force and not _stale(CALLS, [Path(__file__), PKG / "_lib.py"]):
        return CALLS
    src, part = OBJ / f"_calls.{os.getpid()}.c", CALLS.with_suffix(f".{os.getpid()}.tmp")
    try:
        cc = shlex.split(os.environ.get("CC", "")) or [shutil.which("gcc") or "cc"]
        OBJ.mkdir(exist_ok=True)
        src.write_text(_binding_source(sorted(_lib.KINDS, key=_lib.KINDS.get)))
        r = subprocess.run([*cc, "-O2", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], str(src), "-o", str(part)],
                           capture_output=True, text=True)
        why = r.stdout + r.stderr
        if r.returncode == 0 and part.exists():
            os.replace(part, CALLS)
            return CALLS
    except (OSError, ValueError) as e:
        why = str(e)
    finally:
        src.unlink(missing_ok=True)
        part.unlink(missing_ok=True)
    sys.stderr.write(f"{why.rstrip()}\n_calls was not compiled: calls into the libraries go through ctypes, 2 to 3 us slower each\n")
    return None


def _stale(target: Path, deps: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(d.stat().st_mtime > t for d in deps)


def build(force: bool = False, verbose: bool = False, libs: tuple[str, ...] = tuple(LIBS)) -> Path:
    """Compiles what is stale of the named libraries and returns the path of the first one. DJV_NVCC_FLAGS in the
    environment adds flags (e.g. -DDJV_RING_TRACE for the phase stamps of the one-pass MLP kernel; use --force, the
    flag is not part of the staleness check)."""
    nvcc = _nvcc()
    extra = os.environ.get("DJV_NVCC_FLAGS", "").split()
    OBJ.mkdir(exist_ok=True)
    headers = sorted(CSRC.glob("*.cuh")) + sorted((PKG.parent / "include").glob("*.h"))
    wanted = sorted({src for lib in libs for src in sources(lib)})
    jobs = []
    for src in wanted:
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas")
                cmd.insert(2, "-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {cmd[-3]}")
    for lib in libs:
        objs = [OBJ / (s.stem + ".o") for s in sources(lib)]
        if force or _stale(LIBS[lib], objs):
            part = LIBS[lib].with_suffix(f".{os.getpid()}.tmp")
            cmd = [nvcc, "-shared", "-o", str(part), *map(str, objs), "-Xcompiler", "-fPIC", "-lcudart"]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode != 0:
                sys.stderr.write(r.stdout + r.stderr)
                raise RuntimeError("link failed")
            os.replace(part, LIBS[lib])
    build_calls(force)
    return LIBS[libs[0]]


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register / shared-memory usage")
    ap.add_argument("--lib", choices=sorted(LIBS), help="build this library only")
    a = ap.parse_args()
    names = (a.lib,) if a.lib else tuple(LIBS)
    build(force=a.force, verbose=a.verbose, libs=names)
    for name in names:
        print(LIBS[name])
