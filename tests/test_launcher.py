"""The compiled caller of the kernel library: same results as ctypes, and errors instead of wrong calls."""
import ctypes

import pytest

from opaque_b200.ops import lib
from opaque_b200.utils import build


def _toy(tmp_path):
    import importlib.util
    import subprocess
    src = tmp_path / "toy.c"
    src.write_text("""
      #include <stdint.h>
      #include <stdlib.h>
      long long seen[8]; double fseen[4];
      int toy(void* p, int i, long long l, unsigned u, unsigned long long q, float f, double d, const char* s, void* n) {
        seen[0] = (long long)(intptr_t)p; seen[1] = i; seen[2] = l; seen[3] = u; seen[4] = (long long)q; seen[5] = s[1]; seen[6] = n == 0;
        fseen[0] = f; fseen[1] = d; return -7;
      }""")
    so = tmp_path / "libtoy.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    dll = ctypes.CDLL(str(so))
    old_target, old_obj = build.launcher_ext_path, build.OBJ_DIR
    build.launcher_ext_path, build.OBJ_DIR = (lambda: tmp_path / "_launch.so"), tmp_path / "obj"
    try:
        path = build.build_launcher({"toy": "PILUQFDPP"})
        stamp = path.stat().st_mtime_ns
        assert build.build_launcher({"toy": "PILUQFDPP"}) == path and path.stat().st_mtime_ns == stamp      # kept while fresh
    finally:
        build.launcher_ext_path, build.OBJ_DIR = old_target, old_obj
    spec = importlib.util.spec_from_file_location("_launch", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod, dll


def test_arguments_arrive_unchanged(tmp_path):
    mod, dll = _toy(tmp_path)
    good = (2 ** 63 + 5, -3, -2 ** 40, 2 ** 32 - 1, 2 ** 64 - 2, 0.1, 0.1, b"ab", None)
    with pytest.raises(RuntimeError):
        mod.toy(*good)                                            # not bound yet
    mod.bind("toy", ctypes.cast(dll.toy, ctypes.c_void_p).value)
    assert mod.toy(*good) == -7
    seen, fseen = (ctypes.c_longlong * 8).in_dll(dll, "seen"), (ctypes.c_double * 4).in_dll(dll, "fseen")
    assert list(seen)[:7] == [2 ** 63 + 5 - 2 ** 64, -3, -2 ** 40, 2 ** 32 - 1, -2, ord("b"), 1]
    assert fseen[0] == ctypes.c_float(0.1).value and fseen[1] == 0.1
    assert mod.toy(None, True, 0, 0, 0, 1, 2, b"xy", 0) == -7 and fseen[0] == 1.0
    for bad, err in ((good[:-1], TypeError), (("x",) + good[1:], TypeError), (good[:1] + (2 ** 31,) + good[2:], OverflowError),
                     (good[:2] + (2 ** 63,) + good[3:], OverflowError), (good[:5] + ("f",) + good[6:], TypeError)):
        with pytest.raises(err):
            mod.toy(*bad)
    with pytest.raises(KeyError):
        mod.bind("other", 1)


def test_every_launching_entry_point_goes_through_it():
    entries = lib.load()
    sigs = lib.launch_signatures()
    assert set(sigs) | lib._CTYPES_ONLY == set(lib._SIGNATURES)
    for name, sig in sigs.items():
        assert len(sig) == len(lib._SIGNATURES[name]) and type(getattr(entries, name)).__name__ == "builtin_function_or_method"
    # an empty problem returns before anything touches a device
    assert entries.ob_gemm_tn(*[{"P": None, "F": 1.0, "D": 1.0}.get(c, 0) for c in sigs["ob_gemm_tn"]]) == 0


def test_an_installed_extension_needs_no_other_file_and_no_compiler(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "launcher_ext_path", lambda: tmp_path / "_launch.so")
    path = build.build_launcher({"ob_a": "PI"})
    assert {f.name for f in tmp_path.iterdir() if f.suffix != ".lock"} == {"_launch.so"}
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "nowhere")
    monkeypatch.setattr(build, "_find", lambda *a: None)
    assert build.build_launcher({"ob_a": "PI"}) == path
    with pytest.raises(RuntimeError):
        build.build_launcher({"ob_a": "PL"})                      # other signatures: not fresh


def test_an_extension_that_does_not_load_is_built_afresh(tmp_path, monkeypatch):
    def damaged(name):
        path = tmp_path / name
        monkeypatch.setattr(build, "launcher_ext_path", lambda: path)
        data = build.build_launcher({"ob_a": "PI"}).read_bytes()
        path.write_bytes(b"not a library " + data)                # carries the digest all the same
    damaged("_launch.so")
    assert lib._load_launcher({"ob_a": "PI"}).ob_a.__name__ == "ob_a"
    damaged("_launch_2.so")
    monkeypatch.setattr(build, "_find", lambda *a: None)
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert lib._load_launcher({"ob_a": "PI"}) is None
