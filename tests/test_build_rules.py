"""The build rules: an object is compiled again when any file it includes changes."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpfft_b200", "csrc")


def _included(path, seen):
    """Absolute paths of the project files that `path` includes, directly or not."""
    with open(path) as f:
        for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', f.read(), re.M):
            p = os.path.normpath(os.path.join(os.path.dirname(path), name))
            if os.path.exists(p) and p not in seen:
                seen.add(p)
                _included(p, seen)
    return seen


@pytest.mark.skipif(shutil.which("make") is None, reason="no make")
def test_objects_depend_on_every_file_they_include():
    users = {}  # header: objects whose source includes it
    for src in sorted(os.listdir(CSRC)):
        stem, ext = os.path.splitext(src)
        if ext in (".cu", ".cpp"):
            for h in _included(os.path.join(CSRC, src), set()):
                users.setdefault(h, set()).add(stem + ".o")
    assert len(users) >= 10
    for header, objects in users.items():
        # what would be compiled if the header had changed (everything where nothing is built yet)
        out = subprocess.run(["make", "-n", "-C", CSRC, "-W", os.path.relpath(header, CSRC)], check=True,
                             capture_output=True, text=True).stdout
        compiled = set(re.findall(r"-o \S*?(\w+\.o)(?=\s|$)", out))
        assert objects <= compiled, (header, objects - compiled)
