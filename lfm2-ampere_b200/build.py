"""Build liblkb.so (the C-ABI library) in-tree with nvcc for sm_100a.

    python lfm2-ampere_b200/build.py [--force] [--verbose]

nvcc cross-compiles without a GPU.  The library is written next to this file so
that it travels with the source tree; it is never installed into site-packages.
"""
import os
import pathlib
import shlex
import subprocess
import sys
import sysconfig

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE / "csrc"
OUT = HERE / "liblkb.so"
PY_OUT = HERE / ("_fast" + sysconfig.get_config_var("EXT_SUFFIX"))
SOURCES = ["lkb_decode.cu", "lkb_prefill.cu", "lkb_gemm_tc.cu", "lkb_gemm_few.cu", "lkb_fused.cu", "lkb_lmhead.cu", "lkb_mixer.cu", "lkb_pfmix.cu", "lkb_pfattn.cu", "lkb_ep.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC,-fvisibility=hidden", "-Xcompiler", "-O3", "-shared", "-cudart", "static"]


def _older(out, sources):
    return not out.exists() or any(d.stat().st_mtime > out.stat().st_mtime for d in sources + [HERE.parent / "include" / "lkb.h", pathlib.Path(__file__)])


def needs_library():
    return _older(OUT, list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")))


def needs_bindings():
    """Older than their sources, or of another torch (the name has the interpreter's tag)."""
    import torch
    return _older(PY_OUT, list(CSRC.glob("*.cpp"))) or f"torch {torch.__version__};".encode() not in PY_OUT.read_bytes()


def needs_build():
    return needs_library() or needs_bindings()


def build(force=False, verbose=False):
    if force or needs_library():
        srcs = [str(CSRC / s) for s in SOURCES if (CSRC / s).exists()]
        extra = shlex.split(os.environ.get("LKB_NVCC_EXTRA", ""))          # e.g. -DTC_MAGIC=0 while tuning
        cmd = ["nvcc"] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-o", str(OUT)] + srcs + ["-lcuda"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose or r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
        if r.returncode:
            raise RuntimeError("nvcc failed building liblkb.so")
    if force or needs_bindings():
        build_bindings()
    return OUT


def build_bindings():
    """_fast: the CPython bindings of the calls that hosts make most, beside liblkb.so and linked to it."""
    import torch
    from torch.utils import cpp_extension
    inc = [x for p in cpp_extension.include_paths() + [sysconfig.get_paths()["include"]] for x in ("-isystem", p)]
    cmd = ["g++", "-O2", "-std=c++17", "-Wall", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DLKB_BUILT_FOR="torch {torch.__version__};"'] + inc + [
        "-o", str(PY_OUT), str(CSRC / "lkb_py.cpp"), "-L", str(HERE), "-l:liblkb.so", "-Wl,-rpath,$ORIGIN,--disable-new-dtags",      # RPATH: before LD_LIBRARY_PATH
        "-L", str(pathlib.Path(torch.__file__).parent / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError(f"g++ failed building {PY_OUT.name}")


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
