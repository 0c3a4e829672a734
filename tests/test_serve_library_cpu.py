"""The library that a checkout without the full one builds for itself (`make serve`): it links, loads and exports what it promises, and
it is rebuilt when any of its sources changes."""
import os
import re
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = "/usr/local/cuda/bin/nvcc"


def _makefile_objects():
    text = open(os.path.join(ROOT, "Makefile")).read().replace("\\\n", " ")
    return re.findall(r"build/(\w+)\.o", re.search(r"^SERVE_OBJ := (.*)$", text, re.M).group(1))


def test_sources_name_every_object_and_header():
    from llark_b200 import build

    want = set()
    for stem in _makefile_objects():
        want.add(stem + ".cu")
    todo = list(want)
    while todo:
        text = open(os.path.join(build.PKG, "csrc", todo.pop())).read()
        new = set(re.findall(r'#include "(\w+\.cuh?)"', text)) - want
        want |= new
        todo.extend(new)
    assert set(build.SERVE_SOURCES) == want


@pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which("nvcc")), reason="no nvcc")
def test_library_loads(tmp_path):
    so = str(tmp_path / "libllark_serve.so")
    env = dict(os.environ, PATH="/usr/local/cuda/bin:" + os.environ.get("PATH", ""))
    r = subprocess.run(["make", "-j8", "-C", ROOT, so, f"LIB_SERVE={so}"], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    code = ("import sys; from llark_b200 import _lib\n"
            "_lib.LIB_PATH, _lib.SERVE_LIB_PATH = sys.argv[1] + '.none', sys.argv[1]\n"
            "c = _lib.lib()\n"
            "missing = [s for s in _lib.SERVE_SYMBOLS if not hasattr(c, s)]\n"
            "assert c._name == sys.argv[1] and not missing, missing\n")
    env.pop("LLARK_LIB_PATH", None)
    r = subprocess.run([sys.executable, "-c", code, so], cwd=ROOT, env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
