"""The extension's C entries on arguments that they answer without a GPU."""
import ctypes
import os
import subprocess
import sys

import pytest

from autoparallel_b200.ops import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
needs_ext = pytest.mark.skipif(not os.path.exists(build.so_path()), reason="the extension is not built")


def _run(code):
    """In a process of its own: a fault in an entry ends the process."""
    head = "import ctypes, torch\nfrom autoparallel_b200.ops import build\nso = ctypes.CDLL(build.so_path())\n"
    r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    return r.stdout.split()


@needs_ext
def test_slot_workspace_of_an_empty_dispatch():
    """No choices, no tokens, no experts: no workspace, and no division by the empty size."""
    out = _run(
        "f = so.apb_moe_slots_workspace\nf.restype = ctypes.c_longlong\n"
        "print(f(1, 0, 8, 148), f(0, 16, 8, 148), f(1, 16, 0, 148), f(2, 1024, 8, 148) > 0)"
    )
    assert out == ["0", "0", "0", "True"]


@needs_ext
def test_the_extension_brings_no_cxx_library_of_its_own():
    """With a static copy inside, an error with a number in its message ends the process (see ops/build.py)."""
    with open(build.so_path(), "rb") as f:
        assert b"\0libstdc++.so.6\0" in f.read()
