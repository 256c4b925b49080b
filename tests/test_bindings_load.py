"""The native bindings that the package loads: built for this interpreter and this torch, or refused with advice."""
import importlib.util
import os
import pathlib
import shutil
import subprocess
import sys
import sysconfig

import pytest

torch = pytest.importorskip("torch")
PKG = pathlib.Path(__file__).resolve().parent.parent / "lfm2-ampere_b200"
SUFFIX = sysconfig.get_config_var("EXT_SUFFIX")


def _load(path, name, **more):
    spec = importlib.util.spec_from_file_location(name, path, **more)
    mod = importlib.util.module_from_spec(spec)
    sys.modules[name] = mod
    try:
        spec.loader.exec_module(mod)
    finally:
        for k in [k for k in sys.modules if k == name or k.startswith(name + ".")]:
            del sys.modules[k]
    return mod


def _import_copy(tmp_path, put):
    """Import a copy of the package whose bindings `put` provides; the exception it ends with, None without one."""
    pkg = tmp_path / "pkg"
    shutil.copytree(PKG, pkg, ignore=shutil.ignore_patterns("*.so", "csrc", "__pycache__"))
    (pkg / "liblkb.so").symlink_to(PKG / "liblkb.so")
    (tmp_path / "include").mkdir()
    shutil.copy(PKG.parent / "include" / "lkb.h", tmp_path / "include")
    put(pkg)
    try:
        _load(pkg / "__init__.py", "lkb_copy", submodule_search_locations=[str(pkg)])
    except Exception as e:
        return e


def _another_module(pkg):
    """A module that loads, of another build."""
    src = pkg / "other.c"
    src.write_text("#include <Python.h>\nstatic struct PyModuleDef d = {PyModuleDef_HEAD_INIT, \"_fast\", 0, -1};\n"
                   "PyMODINIT_FUNC PyInit__fast(void) { return PyModule_Create(&d); }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], str(src), "-o", str(pkg / ("_fast" + SUFFIX))], check=True)


@pytest.mark.parametrize("put", [lambda pkg: None, lambda pkg: (pkg / ("_fast" + SUFFIX)).write_bytes(b"no library"), _another_module],
                         ids=["missing", "unreadable", "of another build"])
def test_refused_with_advice(tmp_path, put):
    e = _import_copy(tmp_path, put)
    assert type(e).__name__ == "LkbError" and "build.py" in str(e), repr(e)


def test_rebuilt_for_another_torch(tmp_path, monkeypatch):
    """Bindings newer than their sources, but of another torch, are out of date; the library beside them is not."""
    build = _load(PKG / "build.py", "lkb_build_copy")
    data, tag = build.PY_OUT.read_bytes(), torch.__version__.encode()
    assert tag in data and build.PY_OUT.name == "_fast" + SUFFIX
    lib, mod = tmp_path / "liblkb.so", tmp_path / build.PY_OUT.name
    lib.touch()
    mod.write_bytes(data)
    monkeypatch.setattr(build, "OUT", lib)
    monkeypatch.setattr(build, "PY_OUT", mod)
    assert not build.needs_build()
    mod.write_bytes(data.replace(tag, b"0" * len(tag)))
    assert build.needs_build()
    ran = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **k: ran.append(cmd[0]) or subprocess.CompletedProcess(cmd, 0, "", ""))
    build.build()
    assert ran == ["g++"]


def test_one_library_whatever_the_loader_s_path(tmp_path):
    """The bindings call into the library that the package loaded, not into a second copy (never initialised) found on LD_LIBRARY_PATH."""
    shutil.copy(PKG / "liblkb.so", tmp_path)
    code = ("import importlib; importlib.import_module('lfm2-ampere_b200')\n"
            "print({l.split(None, 5)[-1].strip() for l in open('/proc/self/maps') if 'liblkb.so' in l})")
    r = subprocess.run([sys.executable, "-c", code], cwd=PKG.parent, capture_output=True, text=True, check=True, env={**os.environ, "LD_LIBRARY_PATH": str(tmp_path)})
    assert r.stdout.strip() == repr({str(PKG / "liblkb.so")})


def test_build_takes_extra_compiler_options(monkeypatch):
    """LKB_NVCC_EXTRA reaches the compiler that PATH has, between the fixed options and the sources."""
    build = _load(PKG / "build.py", "lkb_build_copy")
    ran = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **k: ran.append(cmd) or subprocess.CompletedProcess(cmd, 0, "", ""))
    monkeypatch.setenv("LKB_NVCC_EXTRA", "-DSOME=1 '-DOTHER=a b'")
    build.build(force=True)
    n = len(build.NVCC_FLAGS)
    assert ran[0][0] == "nvcc" and ran[0][1:n + 1] == build.NVCC_FLAGS and ran[0][n + 1:n + 3] == ["-DSOME=1", "-DOTHER=a b"]
    assert [c[0] for c in ran] == ["nvcc", "g++"]
