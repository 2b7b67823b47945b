"""In-tree native builds: the sm_100a kernel library (nvcc) and the C++ accountant (g++/pybind11).

Artefacts are written next to their sources so they travel with a snapshot of the tree.  A
build is skipped when the artefact is newer than every source; ``force=True`` rebuilds.
"""
from __future__ import annotations

import contextlib
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent.parent
CSRC = PKG / "ops" / "csrc"
KERNEL_LIB = PKG / "ops" / "libopaque_b200.so"
ACC_SRC = PKG / "accounting" / "csrc"

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]
# Approximate division / exp / tanh are fine in the GEMM epilogues and activation kernels.  The translation units that draw
# the DP noise, apply the optimizer, clip materialised gradients and move the experts' rows are compiled WITHOUT them: exponential,
# logarithm, sine / cosine, square roots and divisions are the IEEE-accurate ones and subnormal values are kept.
FAST_MATH = "--use_fast_math"
EXACT_MATH_SOURCES = {"dp_update.cu", "clip_tree.cu", "moe.cu"}
OBJ_DIR = CSRC / "build"


def _find(tool: str, extra: list[str]) -> str | None:
    hit = shutil.which(tool)
    if hit:
        return hit
    for p in extra:
        if os.path.exists(p):
            return p
    return None


@contextlib.contextmanager
def _build_lock(target: Path):
    """Exclusive advisory lock beside ``target`` (held across one compile); a no-op where ``fcntl`` is missing."""
    try:
        import fcntl
    except ImportError:          # pragma: no cover
        yield
        return
    lock_path = target.with_name("." + target.name + ".lock")
    with open(lock_path, "w") as fh:
        fcntl.flock(fh, fcntl.LOCK_EX)
        try:
            yield
        finally:
            fcntl.flock(fh, fcntl.LOCK_UN)


def _stale(target: Path, sources: list[Path]) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(s.stat().st_mtime > t for s in sources)


def _flags_for(src: Path) -> list[str]:
    return list(NVCC_FLAGS) + ([] if src.name in EXACT_MATH_SOURCES else [FAST_MATH])


def build_kernels(force: bool = False, verbose: bool = False) -> Path:
    """Compile every ``.cu`` under ``ops/csrc`` (one object each, rebuilt only when stale) and link one shared library
    for sm_100a."""
    sources = sorted(CSRC.glob("*.cu"))
    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h"))
    deps = sources + headers
    if not force and not _stale(KERNEL_LIB, deps):
        return KERNEL_LIB
    nvcc = _find("nvcc", ["/usr/local/cuda/bin/nvcc"])
    if nvcc is None:
        raise RuntimeError("nvcc not found: cannot build the sm_100a kernel library")
    # Every rank of a job may find the library stale at the same moment: one builds, the others wait on the lock and
    # then see a fresh library.  The output is written under a private name and renamed into place.
    with _build_lock(KERNEL_LIB):
        if not force and not _stale(KERNEL_LIB, deps):
            return KERNEL_LIB
        OBJ_DIR.mkdir(exist_ok=True)
        procs, objs, log = [], [], []
        for src in sources:
            obj = OBJ_DIR / (src.stem + ".o")
            objs.append(obj)
            if force or _stale(obj, [src] + headers):
                cmd = [nvcc, *_flags_for(src), "-c", str(src), "-o", str(obj)]
                if verbose:
                    cmd.insert(1, "-Xptxas=-v")
                procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        failed = []
        for src, obj, proc in procs:                      # the objects compile side by side
            out, _ = proc.communicate()
            log.append(out)
            if proc.returncode != 0:
                obj.unlink(missing_ok=True)
                failed.append(f"{src.name}:\n{out}")
        if failed:
            raise RuntimeError("nvcc failed:\n" + "\n".join(failed))
        tmp = KERNEL_LIB.with_suffix(f".so.tmp{os.getpid()}")
        res = subprocess.run([nvcc, "-shared", "-o", str(tmp), *map(str, objs)], capture_output=True, text=True)
        if res.returncode != 0:
            tmp.unlink(missing_ok=True)
            raise RuntimeError("nvcc link failed:\n" + res.stdout + res.stderr)
        os.replace(tmp, KERNEL_LIB)
    if verbose:
        print("\n".join(log))
    return KERNEL_LIB


def launcher_ext_path() -> Path:
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    return PKG / "ops" / ("_launch" + suffix)


def launcher_source(signatures: dict[str, str]) -> str:
    """C source of the extension that calls the kernel library's entry points.

    ``signatures`` maps an entry point to one letter per argument: ``P`` pointer (an address, ``bytes`` or ``None``), ``I`` int,
    ``L`` long long, ``U`` unsigned, ``Q`` unsigned long long, ``F`` float, ``D`` double.  Every entry point becomes a function
    of the same name that converts its arguments and calls the address handed to ``bind``, without the interpreter lock.
    """
    ctype = {"P": "void*", "I": "int", "L": "long long", "U": "unsigned", "Q": "unsigned long long", "F": "float", "D": "double"}
    out = ["#define PY_SSIZE_T_CLEAN", "#include <Python.h>", "#include <string.h>", """
static int to_ptr(PyObject* o, void** v) {
  if (o == Py_None) { *v = NULL; return 0; }
  if (PyLong_Check(o)) { *v = PyLong_AsVoidPtr(o); return (*v == NULL && PyErr_Occurred()) ? -1 : 0; }
  if (PyBytes_Check(o)) { *v = PyBytes_AS_STRING(o); return 0; }
  PyErr_Format(PyExc_TypeError, "expected an address, bytes or None, got %.80s", Py_TYPE(o)->tp_name);
  return -1;
}
static int to_ll(PyObject* o, long long* v) { *v = PyLong_AsLongLong(o); return (*v == -1 && PyErr_Occurred()) ? -1 : 0; }
static int to_int(PyObject* o, int* v) {
  long long x;
  if (to_ll(o, &x)) return -1;
  if (x < INT_MIN || x > INT_MAX) { PyErr_SetString(PyExc_OverflowError, "argument does not fit an int"); return -1; }
  *v = (int)x;
  return 0;
}
static int to_ull(PyObject* o, unsigned long long* v) { *v = PyLong_AsUnsignedLongLongMask(o); return (*v == (unsigned long long)-1 && PyErr_Occurred()) ? -1 : 0; }
static int to_uint(PyObject* o, unsigned* v) { unsigned long long x; if (to_ull(o, &x)) return -1; *v = (unsigned)x; return 0; }
static int to_double(PyObject* o, double* v) { *v = PyFloat_AsDouble(o); return (*v == -1.0 && PyErr_Occurred()) ? -1 : 0; }
static int to_float(PyObject* o, float* v) { double x; if (to_double(o, &x)) return -1; *v = (float)x; return 0; }
"""]
    conv = {"P": "to_ptr", "I": "to_int", "L": "to_ll", "U": "to_uint", "Q": "to_ull", "F": "to_float", "D": "to_double"}
    for name, sig in signatures.items():
        params = ", ".join(ctype[c] for c in sig)
        out.append(f"static int (*p_{name})({params});")
        out.append(f"static PyObject* w_{name}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{")
        out.append(f'  if (n != {len(sig)}) {{ PyErr_Format(PyExc_TypeError, "{name} takes {len(sig)} arguments, got %zd", n); return NULL; }}')
        out.append(f'  if (p_{name} == NULL) {{ PyErr_SetString(PyExc_RuntimeError, "{name} is not bound"); return NULL; }}')
        for i, c in enumerate(sig):
            out.append(f"  {ctype[c]} v{i}; if ({conv[c]}(a[{i}], &v{i})) return NULL;")
        call = ", ".join(f"v{i}" for i in range(len(sig)))
        out.append(f"  int rc; Py_BEGIN_ALLOW_THREADS rc = p_{name}({call}); Py_END_ALLOW_THREADS")
        out.append("  return PyLong_FromLong(rc);\n}")
    out.append("static PyObject* bind(PyObject* self, PyObject* const* a, Py_ssize_t n) {")
    out.append('  if (n != 2 || !PyUnicode_Check(a[0])) { PyErr_SetString(PyExc_TypeError, "bind(name, address)"); return NULL; }')
    out.append("  const char* s = PyUnicode_AsUTF8(a[0]); void* p; if (s == NULL || to_ptr(a[1], &p)) return NULL;")
    for name in signatures:
        out.append(f'  if (!strcmp(s, "{name}")) {{ *(void**)&p_{name} = p; Py_RETURN_NONE; }}')
    out.append('  PyErr_Format(PyExc_KeyError, "%s", s); return NULL;\n}')
    out.append("static PyMethodDef methods[] = {")
    for name in signatures:
        out.append(f'  {{"{name}", (PyCFunction)(void (*)(void))w_{name}, METH_FASTCALL, NULL}},')
    out.append('  {"bind", (PyCFunction)(void (*)(void))bind, METH_FASTCALL, NULL}, {NULL, NULL, 0, NULL}};')
    out.append('static struct PyModuleDef mod = {PyModuleDef_HEAD_INIT, "_launch", NULL, -1, methods};')
    out.append("PyMODINIT_FUNC PyInit__launch(void) { return PyModule_Create(&mod); }")
    return "\n".join(out) + "\n"


def build_launcher(signatures: dict[str, str], force: bool = False) -> Path:
    """Compile :func:`launcher_source` in-tree.  The extension carries a digest of its source, so an installed copy is fresh
    without any other file; it is rebuilt when the signatures change."""
    target = launcher_ext_path()
    source = launcher_source(signatures)
    mark = "opaque-launch:" + hashlib.sha256(source.encode()).hexdigest()

    def fresh() -> bool:
        return target.exists() and mark.encode() in target.read_bytes()
    if not force and fresh():
        return target
    gcc = _find("gcc", ["/usr/bin/gcc"])
    if gcc is None:
        raise RuntimeError("gcc not found: cannot build the kernel launcher")
    with _build_lock(target):
        if not force and fresh():
            return target
        tmp, tmp_src = target.with_suffix(f".tmp{os.getpid()}"), target.with_suffix(f".tmp{os.getpid()}.c")
        try:
            tmp_src.write_text(source + f'__attribute__((used)) static const char digest[] = "{mark}";\n')
            res = subprocess.run([gcc, "-O2", "-shared", "-fPIC", "-fvisibility=hidden", f"-I{sysconfig.get_paths()['include']}", str(tmp_src),
                                  "-o", str(tmp)], capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError("gcc failed:\n" + res.stdout + res.stderr)
            os.replace(tmp, target)
        finally:
            tmp.unlink(missing_ok=True)
            tmp_src.unlink(missing_ok=True)
    return target


def block_steps_ext_path() -> Path:
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    return PKG / "ops" / ("_blocks" + suffix)


def build_block_steps(force: bool = False) -> Path:
    """Compile ``ops/csrc/block_steps.cpp`` against torch's C++ headers, in-tree.  The extension carries a digest of its sources and of
    torch's version, so an installed copy is fresh without any other file."""
    import torch
    target, sources = block_steps_ext_path(), [CSRC / "block_steps.cpp", CSRC / "api.h"]
    text = torch.__version__ + "".join(p.read_text() for p in sources)
    mark = "opaque-blocks:" + hashlib.sha256(text.encode()).hexdigest()

    def fresh() -> bool:
        return target.exists() and mark.encode() in target.read_bytes()
    if not force and fresh():
        return target
    gxx = _find("g++", ["/usr/bin/g++"])
    if gxx is None:
        raise RuntimeError("g++ not found: cannot build the block steps")
    from torch.utils import cpp_extension
    with _build_lock(target):
        if not force and fresh():
            return target
        tmp = target.with_suffix(f".tmp{os.getpid()}")
        try:
            cuda = Path(_find("nvcc", ["/usr/local/cuda/bin/nvcc"]) or "/usr/local/cuda/bin/nvcc").resolve().parent.parent
            res = subprocess.run(
                [gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                 f'-DOB_DIGEST="{mark}"', *(f"-I{d}" for d in cpp_extension.include_paths()), f"-I{sysconfig.get_paths()['include']}",
                 f"-I{cuda / 'include'}", str(sources[0]), "-o", str(tmp), *(f"-L{d}" for d in cpp_extension.library_paths()),
                 "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"], capture_output=True, text=True)
            if res.returncode != 0:
                raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
            os.replace(tmp, target)
        finally:
            tmp.unlink(missing_ok=True)
    return target


def accounting_ext_path() -> Path:
    suffix = sysconfig.get_config_var("EXT_SUFFIX") or ".so"
    return PKG / "accounting" / ("_native" + suffix)


def build_accounting(force: bool = False) -> Path:
    """Compile the C++17 PLD accountant into a pybind11 extension module."""
    import pybind11
    target = accounting_ext_path()
    sources = sorted(p for p in ACC_SRC.glob("*.cpp") if p.name != "selftest.cpp")     # selftest.cpp has its own main()
    deps = sources + sorted(ACC_SRC.glob("*.hpp"))
    if not sources:
        raise RuntimeError("accounting sources missing")
    if not force and not _stale(target, deps):
        return target
    gxx = _find("g++", ["/usr/bin/g++"])
    if gxx is None:
        raise RuntimeError("g++ not found: cannot build the accountant")
    with _build_lock(target):
        if not force and not _stale(target, deps):
            return target
        tmp = target.with_suffix(f".tmp{os.getpid()}")
        cmd = [gxx, "-O3", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-pthread", "-fopenmp",
               f"-I{pybind11.get_include()}", f"-I{sysconfig.get_paths()['include']}",
               "-o", str(tmp), *map(str, sources)]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            tmp.unlink(missing_ok=True)
            raise RuntimeError("g++ failed:\n" + res.stdout + res.stderr)
        os.replace(tmp, target)
    return target


def build_all(force: bool = False) -> None:
    build_kernels(force)
    from ..ops import lib
    build_launcher(lib.launch_signatures(), force)
    build_block_steps(force)
    build_accounting(force)


if __name__ == "__main__":
    build_all(force="--force" in sys.argv)
    print("built:", KERNEL_LIB, accounting_ext_path())
