"""Runs a piece of Python in a child process whose CUDA runtime is fake_cudart.c: the library's host side, without
a GPU. The code finds `lib` (the library), `fake` (its controls) and `launches()` (kernel names so far) defined."""
import functools
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = r"""
import ctypes, sys
sys.path.insert(0, {root!r})
from wavefd_b200 import _lib
from wavefd_b200.abi import PropagatorABI
lib = _lib.library()
fake = ctypes.CDLL(None)
fake.fake_log.restype = ctypes.c_char_p
fake.fake_live.restype = ctypes.c_long
fake.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
log = lambda what: [l.split()[1:] for l in fake.fake_log().decode().splitlines() if l.startswith(what + " ")]
launches = lambda: [n for n, _ in log("launch")]
def create(name, nx, ny, nz):
    a = PropagatorABI(lib, name)
    dims = (nx, ny, nz, 4, 10.0, 10.0, 10.0, 0.001, 8, 8, nz) if ny else (nx, nz, 4, 10.0, 10.0, 0.001, 8, nz)
    return a, a.alloc(1, 1, *dims)
"""


@functools.lru_cache(maxsize=1)
def _shim():
    out = os.path.join(tempfile.mkdtemp(prefix="fake_cudart_"), "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I/usr/local/cuda/include", "-o", out,
                    os.path.join(HERE, "fake_cudart.c")], check=True)
    return out


def run(code, **env):
    """The child's printed lines."""
    e = {k: v for k, v in os.environ.items() if not k.startswith("WAVEFD_B200_")}
    e.update(env, LD_PRELOAD=_shim())
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT) + code], capture_output=True, text=True, env=e,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout.strip().splitlines()
