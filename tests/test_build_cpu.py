"""What the Makefile and build.py rebuild after an edit, and what holds for all kernels of a kind."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "llark_b200", "csrc")


def _reached(name):
    """The sources under csrc/ that `name` includes, directly or not."""
    todo, seen = [name], set()
    while todo:
        text = open(os.path.join(CSRC, todo.pop())).read()
        new = set(re.findall(r'#include "(\w+\.cuh?)"', text)) - seen
        seen |= new
        todo.extend(new)
    return seen


@pytest.mark.skipif(shutil.which("make") is None, reason="no make")
def test_an_edit_rebuilds_every_object_that_includes_the_file():
    readers = {}
    for src in (n for n in os.listdir(CSRC) if n.endswith(".cu")):
        for header in _reached(src):
            readers.setdefault(header, set()).add(src[:-3])
    assert len(readers) > 3
    for header, want in readers.items():
        r = subprocess.run(["make", "-n", "-C", ROOT, "-W", f"llark_b200/csrc/{header}", "all"], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        assert want <= set(re.findall(r"-o build/(\w+)\.o", r.stdout)), header


@pytest.mark.skipif(shutil.which("make") is None, reason="no make")
def test_native_functions_are_built_for_the_interpreter_that_is_named(tmp_path):
    (tmp_path / "Python.h").write_text("")
    other = tmp_path / "python"
    other.write_text(f"#!/bin/sh\necho {tmp_path} .cpython-399-other.so\n")
    other.chmod(0o755)
    r = subprocess.run(["make", "-n", "-C", ROOT, f"PYTHON={other}", "all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    line, = [x for x in r.stdout.splitlines() if "calls.cpp" in x]
    assert f"-I{tmp_path} " in line and "-o llark_b200/_calls.cpython-399-other.so " in line


@pytest.mark.parametrize("made", [True, False])
def test_a_tree_with_a_library_gets_its_native_functions(tmp_path, monkeypatch, capsys, made):
    import sys

    from llark_b200 import build

    pkg = tmp_path / "llark_b200"
    (pkg / "csrc").mkdir(parents=True)
    (tmp_path / "include").mkdir()
    for f in (pkg / "csrc" / "calls.cpp", tmp_path / "include" / "llark_b200.h", tmp_path / "include" / "Python.h", pkg / "lib.so"):
        f.write_text("")
    monkeypatch.setattr(build, "ROOT", str(tmp_path))
    monkeypatch.setattr(build, "PKG", str(pkg))
    monkeypatch.setattr(build, "FULL", str(pkg / "lib.so"))
    monkeypatch.setattr(build, "_python_h", lambda: str(tmp_path / "include" / "Python.h"))
    monkeypatch.delenv("LLARK_LIB_PATH", raising=False)
    calls = []

    def run(cmd, **kw):
        calls.append(cmd)
        if made:
            open(build.calls_path(), "w").close()
        return subprocess.CompletedProcess(cmd, 0 if made else 2, "", "no compiler")

    monkeypatch.setattr(build.subprocess, "run", run)
    for _ in range(2):
        assert build.ensure_built() == str(pkg / "lib.so")
    assert len(calls) == (1 if made else 2)
    assert f"PYTHON={sys.executable}" in calls[0] and calls[0][-1] == os.path.relpath(build.calls_path(), str(tmp_path))
    assert os.path.basename(build.calls_path()) == "_calls" + build.sysconfig.get_config_var("EXT_SUFFIX")
    assert ("through ctypes" in capsys.readouterr().err) != made


def test_kernels_launched_early_read_no_input_as_read_only():
    """A kernel that lives beside the one before it may not use the loads for memory that nobody writes meanwhile."""
    found = set()
    for name in (n for n in os.listdir(CSRC) if n.endswith(".cu")):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for head, kernel, params, body in re.findall(r"__global__([^;{]*?)\b(\w+_kernel)\(([^{;]*)\)\s*\{(.*?)\n\}", text, re.S):
            if "wait_for_previous()" in body:
                found.add(kernel)
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", params), kernel
                assert not re.search(r"__ldg|ld_ahead|ld\.global\.nc", body), kernel
    assert found == {"rmsnorm_fwd_kernel", "add_rmsnorm_conv4_kernel", "glr_step_kernel", "skinny_kernel", "skinny_tc_kernel"}
