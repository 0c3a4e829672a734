"""What the Makefile and build.py rebuild after an edit."""
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
