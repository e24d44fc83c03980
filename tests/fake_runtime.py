"""Runs a script against the built library on a CUDA runtime without a GPU
(fake_cudart.cpp), in a child process: what the host code allocates, copies and
launches, and what it does when a call fails."""
import os
import subprocess
import sys
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = r"""
import ctypes, sys
import numpy as np
from gdpy import core, inputs
rt = ctypes.CDLL(None)  # the preloaded runtime
rt.fake_log.restype = ctypes.c_char_p
rt.fake_fail.argtypes = [ctypes.c_long]
rt.fake_total.argtypes = [ctypes.c_size_t]
rt.fake_used.restype = ctypes.c_size_t
lib = core.load()
vp = ctypes.c_void_p

def log(clear=True):
    # [(what, address, bytes, stream)]
    out = [l.split() for l in rt.fake_log().decode().splitlines()]
    if clear:
        rt.fake_clear()
    return [(w, int(p, 16) if p != "(nil)" else 0, int(n), int(s, 16) if s != "(nil)" else 0) for w, p, n, s in out]

def ptr(a):
    return a.ctypes.data_as(vp)

def device(n):
    p = vp()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(n)) == 0
    return p
"""


def run(script, env=None):
    with tempfile.TemporaryDirectory() as d:
        so = os.path.join(d, "fake_cudart.so")
        subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include",
                        os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
        e = dict(os.environ, LD_PRELOAD=so, **(env or {}))
        e["PYTHONPATH"] = os.pathsep.join([os.path.join(ROOT, "gfs-dycore_gb300"), HERE, e.get("PYTHONPATH", "")])
        r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=e, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
