"""The build's rules for the two Python extensions (rlx_b200/build.py): what is left out, and when it is built again."""
import os

import pytest

from rlx_b200 import build as B


@pytest.fixture
def calls(monkeypatch):
    seen = []
    monkeypatch.setattr(B, "_build_ext", lambda name, out, flags, ident, force: seen.append((name, ident)))
    return seen


def test_the_library_builds_without_torch(monkeypatch, calls, capsys):
    """A user of the C ABI alone has no torch: the library and CompiledGraph.run's extension are built all the same."""
    monkeypatch.setattr(B.importlib.util, "find_spec", lambda name: None)
    B._build_python_face(False)                                # the step behind the library's own
    assert [n for n, _ in calls] == ["session_ops.cpp"]
    assert "torch" in capsys.readouterr().err


def test_the_library_builds_without_python_headers(monkeypatch, calls, capsys, tmp_path):
    monkeypatch.setattr(B.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    B._build_python_face(False)
    assert calls == [] and "Python.h" in capsys.readouterr().err


def test_extensions_are_built_again_for_another_torch_or_interpreter(monkeypatch, calls, tmp_path):
    B._build_python_face(False)
    ident = dict(calls)
    assert set(ident) == {"session_ops.cpp", "torch_ops.cpp"}
    src, out = tmp_path / "a.cpp", tmp_path / "_a.so"
    src.write_text("")
    out.write_text("")
    monkeypatch.setattr(B, "OBJ", str(tmp_path))
    assert not B._ext_is_current(str(out), [str(src)], "one")             # nobody noted what it was built for
    (tmp_path / "_a.so.for").write_text("one")
    assert B._ext_is_current(str(out), [str(src)], "one") and not B._ext_is_current(str(out), [str(src)], "two")
    os.utime(src, (os.path.getmtime(out) + 5,) * 2)
    assert not B._ext_is_current(str(out), [str(src)], "one")
    # another version, another place, another interpreter: another note
    root, before = B._torch_root(), B._built_for(B._torch_root())
    assert B._built_for("/elsewhere/torch") != before
    monkeypatch.setattr(B.importlib.metadata, "version", lambda name: "0.0")
    assert B._built_for(root) != before
    monkeypatch.setattr(B.sys, "version", "another")
    assert B._built_for(None) != ident["session_ops.cpp"]


def test_the_build_runs_before_there_is_a_library(tmp_path):
    """The command that the import error names does not itself import the package, which needs the library."""
    import shutil
    import subprocess
    import sys
    pkg = tmp_path / "rlx_b200"
    shutil.copytree(B.PKG, pkg, ignore=shutil.ignore_patterns("*.so", "csrc", "__pycache__"))
    r = subprocess.run([sys.executable, "-c", "import rlx_b200"], cwd=tmp_path, capture_output=True, text=True)
    command = r.stderr.split("build it with `")[1].split("`")[0].split()
    assert r.returncode and command[0] == "python"
    r = subprocess.run([sys.executable, *command[1:]], cwd=tmp_path, capture_output=True, text=True, env={**os.environ, "NVCC": "", "PATH": ""})
    assert "ImportError" not in r.stderr and "missing: build it" not in r.stderr, r.stderr


def test_dependent_kernels_read_no_invariant_parameters():
    """A kernel that is launched as a programmatic dependent starts while the one in front still writes its inputs.  Memory behind a
    `const __restrict__` parameter may be read ahead of griddep_wait(): only the weights may be one."""
    import glob
    import re
    kernels = 0
    for path in sorted(glob.glob(os.path.join(B.PKG, "csrc", "**", "*.cu"), recursive=True)):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)?(\w+)\(([^{]*)\)\s*\{(.*?)\n\}", text, re.S):
            if "griddep_wait()" not in m[3]:
                continue
            kernels += 1
            invariant = set(re.findall(r"const\s+[\w ]+\*\s*__restrict__\s+(\w+)", m[2])) - {"w"}
            assert not invariant, (os.path.basename(path), m[1], invariant)
    assert kernels >= 15
