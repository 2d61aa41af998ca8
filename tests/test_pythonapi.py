"""The renderer's use of the Python C API: the function objects of
ctypes.pythonapi belong to the whole process, so the package neither sets
their prototypes nor depends on what others set."""

import subprocess
import sys
from pathlib import Path

ROOT = str(Path(__file__).resolve().parent.parent)

IMPORT_LEAVES_PROTOTYPES = """
import ctypes
api = ctypes.pythonapi
before = [(f.argtypes, f.restype) for f in (api.PyBytes_FromStringAndSize, api.PyBytes_AsString)]
import pyvr_gb300.renderer
assert [(f.argtypes, f.restype) for f in (api.PyBytes_FromStringAndSize, api.PyBytes_AsString)] == before
"""

OTHERS_PROTOTYPES_DO_NOT_MATTER = """
import ctypes
import pyvr_gb300.renderer as r
api = ctypes.pythonapi
api.PyBytes_FromStringAndSize.argtypes = [ctypes.c_void_p, ctypes.c_ssize_t]
api.PyBytes_FromStringAndSize.restype = ctypes.c_void_p
api.PyBytes_AsString.restype = ctypes.c_char_p
out = r._bytes_new(None, 300)
assert type(out) is bytes and len(out) == 300
p = r._bytes_address(out)
assert type(p) is int
ctypes.memset(p, 7, 300)
assert out == b"\\x07" * 300
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_import_leaves_the_prototypes_alone():
    _run(IMPORT_LEAVES_PROTOTYPES)


def test_prototypes_set_elsewhere_do_not_matter():
    _run(OTHERS_PROTOTYPES_DO_NOT_MATTER)
