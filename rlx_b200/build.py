"""Builds rlx_b200/librlxq.so (the C-ABI library) with nvcc for sm_100a, in-tree, and rlx_b200/_torch_ops.so, the
native form of the Python calls on torch tensors, with the host compiler.

    python rlx_b200/build.py [--force] [--verbose]

Only nvcc is needed (no GPU): the objects are cross-compiled.  Objects are cached under
rlx_b200/csrc/build/ and rebuilt when a source or header is newer, the extensions also when the interpreter or torch is
another one than they were built for.  The extensions are left out where Python's headers or torch are missing.
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(PKG, "librlxq.so")
OPS = os.path.join(PKG, "_torch_ops.so")
SESSION_OPS = os.path.join(PKG, "_session_ops.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the rlxq library cannot be built")


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "host", "*.cu")))


def _headers() -> list[str]:
    return (glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) +
            glob.glob(os.path.join(CSRC, "host", "*.h*")) +
            glob.glob(os.path.join(PKG, "..", "include", "*.h")))


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJ, os.path.relpath(src, CSRC).replace(os.sep, "_")[:-3] + ".o")
    cmd = [_nvcc(), *NVCC_FLAGS, "-I", os.path.join(PKG, "..", "include"), "-I", CSRC, "-c", src, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)
    return obj


def _torch_root() -> str | None:
    """Where torch is installed, without importing it; None where it is not."""
    try:
        spec = importlib.util.find_spec("torch")
    except (ImportError, ValueError):
        return None
    root = os.path.dirname(spec.origin) if spec and spec.origin else None
    return root if root and os.path.isdir(os.path.join(root, "include")) else None


def _python_include() -> str | None:
    inc = sysconfig.get_paths()["include"]
    return inc if os.path.exists(os.path.join(inc, "Python.h")) else None


def _built_for(torch_root: str | None) -> str:
    """What an extension is built for: this interpreter and, with torch_root, this torch."""
    ident = f"{sys.version} {sysconfig.get_config_var('SOABI')} {_python_include()}"
    if torch_root:
        try:
            ident += f" torch {importlib.metadata.version('torch')} {torch_root}"
        except importlib.metadata.PackageNotFoundError:
            ident += f" torch {torch_root}"
    return ident


def _ext_is_current(out: str, sources, ident: str) -> bool:
    """Whether `out` is newer than its sources and was built for `ident` (its note lies with the objects)."""
    note = os.path.join(OBJ, os.path.basename(out) + ".for")
    if not (os.path.exists(out) and os.path.exists(note)) or os.path.getmtime(out) < max(os.path.getmtime(p) for p in sources):
        return False
    with open(note) as f:
        return f.read() == ident


def _build_ext(name: str, out: str, flags, ident: str, force: bool) -> None:
    """csrc/python/<name> against this interpreter and librlxq.so beside it; flags() -> what else it needs."""
    src = os.path.join(CSRC, "python", name)
    if not force and _ext_is_current(out, [src, *glob.glob(os.path.join(PKG, "..", "include", "*.h"))], ident):
        return
    compile_flags, link_flags = flags()
    cmd = [os.environ.get("CXX") or shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           *compile_flags, "-isystem", _python_include(), "-I", os.path.join(PKG, "..", "include"), src, "-o", out,
           *link_flags, "-L", PKG, "-l:librlxq.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed for {src}:\n{r.stdout}\n{r.stderr}")
    with open(os.path.join(OBJ, os.path.basename(out) + ".for"), "w") as f:
        f.write(ident)


def _torch_flags():
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    return ([f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             "-isystem", os.path.join(root, "include"), "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"),
             "-isystem", os.path.join(cuda, "include")],
            ["-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"])


def _build_python_face(force: bool) -> None:
    """The two extensions.  A user of the C ABI alone needs neither: without Python's headers none is built, without torch only
    CompiledGraph.run's.  The calls that need a missing one say so when they are made."""
    if _python_include() is None:
        sys.stderr.write("rlx_b200: no Python.h, librlxq.so is built without the Python extensions\n")
        return
    _build_ext("session_ops.cpp", SESSION_OPS, lambda: ([], []), _built_for(None), force)
    root = _torch_root()
    if root is None:
        sys.stderr.write("rlx_b200: torch is not installed, librlxq.so is built without _torch_ops.so\n")
        return
    _build_ext("torch_ops.cpp", OPS, _torch_flags, _built_for(root), force)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = sources()
    newest_hdr = max((os.path.getmtime(h) for h in _headers()), default=0.0)
    todo, objs = [], []
    for s in srcs:
        obj = os.path.join(OBJ, os.path.relpath(s, CSRC).replace(os.sep, "_")[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(s), newest_hdr):
            todo.append(s)
    if todo:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(todo))) as ex:
            list(ex.map(lambda s: _compile(s, verbose), todo))
    if todo or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
               "-lcudart", "-ldl", "-lpthread"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_python_face(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
