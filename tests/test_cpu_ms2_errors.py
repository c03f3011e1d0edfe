"""What the MS2 reader cannot take comes back as a status, never as a C++ exception through the
C interface (which ends the process, so each call runs in one of its own)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

READ = """
import ctypes as C, resource, sys
from hicops_gb300 import _lib
lib = _lib.load()
resource.setrlimit(resource.RLIMIT_AS, (1 << 33, 1 << 33))
h, n, m = C.c_void_p(), C.c_uint32(), C.c_uint32()
print(lib.hc_ms2_read(sys.argv[1].encode(), 100, C.byref(h), C.byref(n), C.byref(m)), h.value)
"""


@pytest.mark.parametrize("what,status", [("larger than memory", -3007), ("directory", -3013), ("missing", -3013),
                                         ("empty", -3004)])
def test_read_returns_a_status(what, status, tmp_path):
    from hicops_gb300 import build as B
    B.build(quiet=True)
    path = tmp_path / "x.ms2"
    if what == "directory":
        path.mkdir()
    elif what != "missing":
        path.write_bytes(b"")
        if what != "empty":
            os.truncate(path, 1 << 34)  # a hole
    r = subprocess.run([sys.executable, "-c", READ, str(path)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == [str(status), "None"], (r.returncode, r.stdout, r.stderr[-500:])
