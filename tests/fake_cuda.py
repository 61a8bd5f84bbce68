"""Runs Python code with the library on the fake CUDA runtime
(tests/cpp/fake_cudart.cpp) in front of the real one, in a process of its own,
so that host code is tested on machines without a GPU."""
import os
import subprocess
import sys
import textwrap

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)

PRELUDE = """
import ctypes, os, sys
sys.path[:0] = [%r, %r]
import numpy as np
import b200dwf
lib = b200dwf.lib()
fake = ctypes.CDLL(%r)
fake.fake_log.restype = ctypes.c_char_p
fake.fake_used.restype = fake.fake_pool_idle.restype = ctypes.c_size_t
fake.fake_limit.argtypes = [ctypes.c_size_t]
fake.fake_pointer.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]
def log():
    out = fake.fake_log().decode().splitlines()
    fake.fake_clear()
    return out
def array(n, offset=0):
    '''n doubles `offset` doubles behind a 64-byte boundary, and their address'''
    a = np.zeros(n + offset + 8)
    k = (-(a.ctypes.data // 8)) %% 8 + offset
    a = a[k:k + n]
    return a, ctypes.c_void_p(a.ctypes.data)
lat = (ctypes.c_int * 4)(4, 4, 4, 4)
nlink = 72 * 256
HOST, DEVICE, MANAGED = 1, 2, 3
"""


def run(tmp_path, code, **env):
    so = str(tmp_path / "fake_cudart.so")
    if not os.path.exists(so):
        subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", "/usr/local/cuda/include",
                        os.path.join(HERE, "cpp", "fake_cudart.cpp"), "-o", so, "-ldl"], check=True)
    src = PRELUDE % (REPO, os.path.join(REPO, "lqcd-dwf-hmc_b200"), so) + textwrap.dedent(code)
    r = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=so, B200_AUTOTUNE="0", **env))
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
