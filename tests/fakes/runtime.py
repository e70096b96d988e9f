"""Runs a piece of Python on a fake CUDA runtime (cuda_two_devices.cpp), in a process of its own."""
import os
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent.parent

# what the pieces have: the fake, the library under it, ``p`` for any device array, and a check of a status
OPENING = r"""
import ctypes as C, sys
fake, lib = C.CDLL(sys.argv[1]), C.CDLL(sys.argv[2])
from gisapr_gb300 import _native as nat
for name, args in nat.SIGNATURES.items():
    getattr(lib, name).argtypes = args
lib.gisapr_last_error.restype = C.c_char_p
memory = C.create_string_buffer(1 << 20)
p = C.c_void_p((C.addressof(memory) + 255) & ~255)
def ok(rc, what):
    assert rc == 0, (what, lib.gisapr_last_error())
"""


def run_on_fake(code, tmp_path) -> str:
    """The output of ``code`` on the fake runtime; an error there is a failure here."""
    from gisapr_gb300 import _native
    from gisapr_gb300.build_native import cuda_home
    fake = tmp_path / "libfake.so"
    r = subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", str(cuda_home() / "include"), "-o", str(fake),
                        str(HERE / "cuda_two_devices.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([sys.executable, "-c", OPENING + code, str(fake), str(_native.LIB_PATH)],
                       env=dict(os.environ, LD_PRELOAD=str(fake), PYTHONPATH=str(ROOT)), cwd=str(ROOT),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
