"""In-tree build of the native libraries.

Three shared objects are produced next to the package (never installed into
site-packages, so a process that loads them shows the in-tree path):

* ``prometheus_b200/_lib/libpb200_kernels.so`` — every ``csrc/kernels/*.cu`` and
  ``csrc/comm/*.cu`` compiled by ``nvcc`` for ``sm_100a`` only. The kernels
  export a plain C ABI (raw device pointers + a stream handle) and are bound
  with ``ctypes``; nothing in them depends on the PyTorch headers, so a file
  compiles in seconds.
* ``prometheus_b200/_lib/_pb200_call*.so`` — typed callers for those symbols' signatures,
  generated from their declarations in ``ops/_lib.py``: what a launch from Python goes through.
* ``prometheus_b200/_lib/_pb200_native*.so`` — the C++17 systems code under
  ``csrc/native`` (checkpoint store, data loader, controller, observability,
  harness) bound with pybind11.

``python -m prometheus_b200._build`` builds all; ``build_all()`` is what
``__graft_entry__.build()`` calls. Objects are rebuilt only when their source
(or a shared header) is newer.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "csrc"
LIB_DIR = Path(__file__).resolve().parent / "_lib"
OBJ_DIR = ROOT / "build" / "obj"

KERNEL_LIB = LIB_DIR / "libpb200_kernels.so"
NVCC_ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC",
              "-Xcompiler", "-fvisibility=hidden"]


SANITIZE_ENV = "PB200_NATIVE_SANITIZE"     # "", "address,undefined" or "thread": which build to load


def _san_tag(sanitize: str | None) -> str:
    return "" if not sanitize else "_" + sanitize.replace(",", "_")


def native_lib_path(sanitize: str | None = None) -> Path:
    """The pybind11 module; with ``sanitize`` (default: the ``PB200_NATIVE_SANITIZE``
    environment variable) the instrumented build that lives beside it in ``_lib/san_*``."""
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    sanitize = os.environ.get(SANITIZE_ENV, "") if sanitize is None else sanitize
    if sanitize:
        return LIB_DIR / ("san" + _san_tag(sanitize)) / f"_pb200_native{suffix}"
    return LIB_DIR / f"_pb200_native{suffix}"


def sanitizer_runtime(sanitize: str) -> str:
    """Path of the sanitizer runtime to ``LD_PRELOAD`` when an instrumented module is loaded
    into an uninstrumented interpreter."""
    lib = "libtsan.so" if "thread" in sanitize else "libasan.so"
    # libstdc++ rides along: the interpreter is not linked against it, and the runtime resolves
    # its __cxa_throw interceptor when it starts
    paths = [subprocess.run(["gcc", f"-print-file-name={name}"], capture_output=True, text=True).stdout.strip()
             for name in (lib, "libstdc++.so")]
    return " ".join(paths)


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found")


def _newer(src_list, target: Path) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(s).stat().st_mtime > t for s in src_list)


def _run(cmd, verbose=False):
    if verbose:
        print(" ".join(str(c) for c in cmd), flush=True)
    r = subprocess.run([str(c) for c in cmd], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"build failed: {' '.join(str(c) for c in cmd)}\n{r.stdout}\n{r.stderr}")
    return r.stdout + r.stderr


def kernel_sources() -> list[Path]:
    return sorted(list((CSRC / "kernels").glob("*.cu")) + list((CSRC / "comm").glob("*.cu")))


def build_kernels(verbose: bool = False, force: bool = False, debug_bounds: bool = False) -> Path:
    """Compile every .cu for sm_100a and link libpb200_kernels.so. ``debug_bounds`` builds
    ``libpb200_kernels_dbg.so`` with ``-DPB_DEBUG_BOUNDS`` instead: indices that come from data
    are checked in the kernels and a violation is recorded and skipped rather than executed
    (``PB200_DEBUG_BOUNDS=1`` makes the package load that library)."""
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    nvcc = _nvcc()
    tag = "dbg_" if debug_bounds else ""
    extra = ["-DPB_DEBUG_BOUNDS"] if debug_bounds else []
    target = LIB_DIR / "libpb200_kernels_dbg.so" if debug_bounds else KERNEL_LIB
    headers = list((CSRC / "kernels").glob("*.cuh")) + list((CSRC / "comm").glob("*.cuh"))
    srcs = kernel_sources()
    objs, jobs = [], []
    for src in srcs:
        obj = OBJ_DIR / (tag + src.parent.name + "_" + src.stem + ".o")
        objs.append(obj)
        if force or _newer([src, *headers], obj):
            jobs.append([nvcc, *NVCC_ARCH, *NVCC_FLAGS, *extra, "-rdc=false", "-I", CSRC / "kernels", "-I",
                         CSRC / "comm", "-c", src, "-o", obj])
    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(lambda c: _run(c, verbose), jobs))
    if force or jobs or _newer(objs, target):
        # link beside the target and rename: a process (or a snapshot of the tree) never sees a
        # half-written library
        tmp = target.with_name(target.name + ".tmp")
        _run([nvcc, *NVCC_ARCH, "-shared", "-o", tmp, *objs], verbose)
        os.replace(tmp, target)
    return target


def build_native(verbose: bool = False, force: bool = False, sanitize: str = "") -> Path | None:
    """Compile csrc/native/*.cpp into the pybind11 module (host only, no CUDA).

    ``sanitize`` = ``"address,undefined"`` or ``"thread"`` builds an instrumented copy
    (``-fsanitize=...``, ``-O1 -g``, frame pointers kept) under ``_lib/san_*`` for the host-side
    race / memory checks of the systems code (the asynchronous checkpoint writer, the loader):
    load it with ``PB200_NATIVE_SANITIZE=<same string>`` and the matching runtime preloaded
    (``sanitizer_runtime``)."""
    srcs = sorted((CSRC / "native").glob("*.cpp"))
    if not srcs:
        return None
    import pybind11

    if sanitize not in ("", "address,undefined", "thread"):
        raise ValueError("sanitize must be '', 'address,undefined' or 'thread'")
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    headers = [h for pat in ("*.hpp", "*.h", "*.inc") for h in (CSRC / "native").glob(pat)]
    inc = ["-I", pybind11.get_include(), "-I", sysconfig.get_paths()["include"],
           "-I", CSRC / "native"]
    flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", "-Wno-unused-function"]
    link_extra = []
    if sanitize:
        flags = ["-O1", "-g", "-fno-omit-frame-pointer", f"-fsanitize={sanitize}", "-std=c++17", "-fPIC",
                 "-fvisibility=hidden", "-Wall", "-Wno-unused-function"]
        link_extra = [f"-fsanitize={sanitize}"]
    objs, jobs = [], []
    for src in srcs:
        obj = OBJ_DIR / ("native" + _san_tag(sanitize) + "_" + src.stem + ".o")
        objs.append(obj)
        if force or _newer([src, *headers], obj):
            jobs.append(["g++", *flags, *inc, "-c", src, "-o", obj])
    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(lambda c: _run(c, verbose), jobs))
    out = native_lib_path(sanitize)
    out.parent.mkdir(parents=True, exist_ok=True)
    if force or jobs or _newer(objs, out):
        tmp = out.with_name(out.name + ".tmp")
        _run(["g++", "-shared", "-o", tmp, *objs, *link_extra, "-lpthread", "-lz"], verbose)
        os.replace(tmp, out)
    return out


CALL_CPP_HEAD = r"""// Generated from the signatures of prometheus_b200/ops/_lib.py: one typed caller per distinct signature.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <cstring>
namespace {
bool get(PyObject* o, void*& v) {
  if (o == Py_None) { v = nullptr; return true; }
  if (!PyLong_Check(o)) { PyErr_SetString(PyExc_TypeError, "a device pointer is an int or None"); return false; }
  v = reinterpret_cast<void*>(PyLong_AsUnsignedLongLongMask(o));
  return !PyErr_Occurred();
}
// integers as a foreign call takes them: anything with an index, cut to the width of the argument
bool get(PyObject* o, long& v) {
  int wide = 0;
  v = PyLong_AsLongAndOverflow(o, &wide);
  if (wide) v = static_cast<long>(PyLong_AsUnsignedLongLongMask(o));
  return !(v == -1 && PyErr_Occurred());
}
bool get(PyObject* o, int& v) { long l; if (!get(o, l)) return false; v = static_cast<int>(l); return true; }
bool get(PyObject* o, float& v) {
  const double d = PyFloat_AsDouble(o);
  v = static_cast<float>(d);
  return !(d == -1.0 && PyErr_Occurred());
}
template <typename... A> struct Caller {
  template <size_t... I>
  static PyObject* run(PyObject* self, PyObject* const* a, std::index_sequence<I...>) {
    std::tuple<A...> v;
    if (!(get(a[I], std::get<I>(v)) && ...)) return nullptr;
    const auto fn = reinterpret_cast<int (*)(A...)>(PyCapsule_GetPointer(self, nullptr));
    int rc;
    Py_BEGIN_ALLOW_THREADS   // as a foreign call does: a full launch queue must not hold up other threads
    rc = fn(std::get<I>(v)...);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
  }
  static PyObject* call(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    if (n != static_cast<Py_ssize_t>(sizeof...(A))) {
      PyErr_Format(PyExc_TypeError, "%zd arguments, %zd expected", n, static_cast<Py_ssize_t>(sizeof...(A)));
      return nullptr;
    }
    return run(self, a, std::index_sequence_for<A...>{});
  }
};
struct Entry { const char* sig; PyMethodDef def; };
"""

CALL_CPP_TAIL = r"""
// bind(address, signature): a callable for the exported function at that address, or None
PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long addr;
  const char* sig;
  if (!PyArg_ParseTuple(args, "Ks", &addr, &sig)) return nullptr;
  for (Entry& e : entries)
    if (std::strcmp(e.sig, sig) == 0) {
      PyObject* cap = PyCapsule_New(reinterpret_cast<void*>(addr), nullptr, nullptr);
      if (cap == nullptr) return nullptr;
      PyObject* f = PyCFunction_New(&e.def, cap);
      Py_DECREF(cap);
      return f;
    }
  Py_RETURN_NONE;
}
PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_pb200_call", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
}  // namespace
PyMODINIT_FUNC PyInit__pb200_call() { return PyModule_Create(&module); }
"""


def call_lib_path() -> Path:
    return LIB_DIR / f"_pb200_call{sysconfig.get_config_var('EXT_SUFFIX') or '.so'}"


def build_call(verbose: bool = False, force: bool = False) -> Path:
    """The launch path's binding: typed callers for the signatures declared in ``ops/_lib.py`` (read
    from its source, nothing is imported). Converting the 27 arguments of a matrix product through
    ctypes took as long as launching it."""
    import ast

    src = Path(__file__).resolve().parent / "ops" / "_lib.py"
    tree = ast.parse(src.read_text())
    table = next(n.value for n in tree.body if isinstance(n, ast.Assign) and getattr(n.targets[0], "id", "") == "_SIGS")
    sigs = sorted({"".join(e.id for e in v.elts) for v in table.values})
    types = {"P": "void*", "I": "int", "L": "long", "F": "float"}
    rows = ",\n".join(f'    {{"{s}", {{"{s or "none"}", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>('
                      f'Caller<{", ".join(types[c] for c in s)}>::call)), METH_FASTCALL, nullptr}}}}' for s in sigs)
    head = CALL_CPP_HEAD.replace("#include <cstring>", "#include <cstring>\n#include <tuple>\n#include <utility>")
    text = head + "Entry entries[] = {\n" + rows + "};\n" + CALL_CPP_TAIL
    LIB_DIR.mkdir(parents=True, exist_ok=True)
    OBJ_DIR.mkdir(parents=True, exist_ok=True)
    cpp, out = OBJ_DIR / "pb200_call.cpp", call_lib_path()
    if force or not cpp.exists() or cpp.read_text() != text or _newer([cpp], out):
        cpp.write_text(text)
        tmp = out.with_name(out.name + ".tmp")
        _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall",
              "-I", sysconfig.get_paths()["include"], cpp, "-o", tmp], verbose)
        os.replace(tmp, out)
    return out


def build_all(verbose: bool = False, force: bool = False) -> None:
    build_call(verbose, force)
    build_kernels(verbose, force)
    build_kernels(verbose, force, debug_bounds=True)     # the self-checking variant rides along
    build_native(verbose, force)


if __name__ == "__main__":
    san = [a.split("=", 1)[1] for a in sys.argv if a.startswith("--sanitize=")]
    if "--debug-bounds" in sys.argv:
        print("built:", build_kernels(verbose="-v" in sys.argv, force="--force" in sys.argv, debug_bounds=True))
    elif san:
        print("built:", build_native(verbose="-v" in sys.argv, force="--force" in sys.argv, sanitize=san[0]))
    else:
        build_all(verbose="-v" in sys.argv, force="--force" in sys.argv)
        print("built:", KERNEL_LIB, native_lib_path(""))
