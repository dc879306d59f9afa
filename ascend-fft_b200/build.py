"""Build libbfly_b200.so in-tree for sm_100a.

CUDA translation units are compiled by nvcc with `-gencode arch=compute_100a,code=sm_100a`,
host units by g++, and everything is linked into bfly/_lib/libbfly_b200.so next to the Python
package (the CUDA runtime is linked statically); csrc_torch/ becomes the Python module
bfly/_lib/_torch_ops.so on top of it where torch is installed (the library itself needs none).
Objects go to _build/; a unit is rebuilt only when it or a header is newer than its object, the module
also when it was built for another torch or Python.

    python ascend-fft_b200/build.py [--force] [--jobs N]
"""
from __future__ import annotations

import argparse
import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
ROOT = PKG.parent
CSRC = PKG / "csrc"
BUILD = PKG / "_build"
LIBDIR = PKG / "bfly" / "_lib"
LIB = LIBDIR / "libbfly_b200.so"
TORCH_SRC = PKG / "csrc_torch" / "torch_ops.cpp"
TORCH_LIB = LIBDIR / "_torch_ops.so"   # the Python module bfly/ops.py calls

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
INCLUDES = ["-I", str(ROOT / "include"), "-I", str(CSRC)]


def nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (CUDA 12.9 toolkit required)")


def sources():
    cu = sorted(CSRC.glob("*.cu"))
    cpp = sorted(CSRC.glob("*.cpp"))
    return cu, cpp


def headers():
    return list(CSRC.glob("*.h")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.hpp")) + \
        list((ROOT / "include").rglob("*.h*"))


def stale(src: Path, obj: Path, deps) -> bool:
    if not obj.exists():
        return True
    t = obj.stat().st_mtime
    return src.stat().st_mtime > t or any(h.stat().st_mtime > t for h in deps)


def compile_one(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("compile failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stderr


def torch_abi() -> str | None:
    """What the torch module is built against; None without torch."""
    import importlib.metadata
    import sysconfig
    try:
        return f"torch {importlib.metadata.version('torch')} {sysconfig.get_config_var('SOABI')}"
    except importlib.metadata.PackageNotFoundError:
        return None


def torch_cmd(obj: Path):
    """Compile and link commands of the torch module (C++ against the installed torch)."""
    import sysconfig

    from torch.utils import cpp_extension
    includes = [*INCLUDES, "-I", sysconfig.get_paths()["include"], "-I", str(Path(nvcc()).parents[1] / "include")]
    for d in cpp_extension.include_paths():
        includes += ["-isystem", d]
    dirs = cpp_extension.library_paths()
    return (["g++", "-std=c++17", "-O2", "-fPIC", "-Wall", "-Wextra", f"-DTORCH_EXTENSION_NAME={TORCH_LIB.stem}",
             *includes, "-c", str(TORCH_SRC), "-o", str(obj)],
            ["g++", "-shared", "-o", str(TORCH_LIB.with_suffix(".so.tmp")), str(obj), *[f"-L{d}" for d in dirs],
             f"-L{LIBDIR}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", f"-l:{LIB.name}",
             "-Wl,-rpath,$ORIGIN"])


def build_torch_object(force: bool):
    """Compile the torch module where it is stale; its link command where that has to run."""
    abi = torch_abi()
    if abi is None:
        print("torch is not installed: the module of bfly's torch functions is not built", file=sys.stderr)
        return None
    obj, stamp = BUILD / (TORCH_SRC.stem + ".torch.o"), BUILD / (TORCH_SRC.stem + ".torch.abi")
    fresh = stamp.exists() and stamp.read_text() == abi and not force and \
        not stale(TORCH_SRC, obj, [ROOT / "include" / "bfly_b200.h"])
    if fresh and TORCH_LIB.exists() and TORCH_LIB.stat().st_mtime >= obj.stat().st_mtime:
        return None
    compile_cmd, link_cmd = torch_cmd(obj)
    if not fresh:
        stamp.unlink(missing_ok=True)
        compile_one(compile_cmd)
        stamp.write_text(abi)
    return link_cmd


def build(force: bool = False, jobs: int | None = None, verbose: bool = False) -> Path:
    BUILD.mkdir(parents=True, exist_ok=True)
    LIBDIR.mkdir(parents=True, exist_ok=True)
    cu, cpp = sources()
    deps = headers()
    cmds, objs = [], []
    for src in cu:
        obj = BUILD / (src.stem + ".o")
        objs.append(obj)
        if force or stale(src, obj, deps):
            cmds.append([nvcc(), "-std=c++17", "-O3", "-lineinfo", *ARCH, "-Xcompiler", "-fPIC",
                         "-Xptxas", "-v" if verbose else "-O3", *INCLUDES, "-c", str(src), "-o", str(obj)])
    for src in cpp:
        obj = BUILD / (src.stem + ".o")
        objs.append(obj)
        if force or stale(src, obj, deps):
            cmds.append(["g++", "-std=c++17", "-O2", "-fPIC", "-Wall", "-Wextra", *INCLUDES,
                         "-c", str(src), "-o", str(obj)])
    workers = jobs or min(len(cmds) + 1, os.cpu_count() or 4)
    with cf.ThreadPoolExecutor(max_workers=workers) as ex:
        module = ex.submit(build_torch_object, force)   # the longest of them
        for out in ex.map(compile_one, cmds):
            if verbose and out:
                print(out, file=sys.stderr)
        if cmds or not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
            tmp = LIB.with_suffix(".so.tmp")
            compile_one([nvcc(), "-shared", *ARCH, "-cudart", "static", "-o", str(tmp),
                         *[str(o) for o in objs], "-lpthread", "-ldl", "-lrt"])
            os.replace(tmp, LIB)
        link = module.result()
    if link:
        compile_one(link)
        os.replace(TORCH_LIB.with_suffix(".so.tmp"), TORCH_LIB)
    return LIB


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--jobs", type=int, default=None)
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args(argv)
    print(build(a.force, a.jobs, a.verbose))


if __name__ == "__main__":
    main()
