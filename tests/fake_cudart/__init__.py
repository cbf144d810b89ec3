"""The CUDA runtime without a device (fake_cudart.cpp), built and put in front
of libcudart for one Python program: ``run(text)`` runs `text` after the lines
of PRELUDE and returns what it prints."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
SRC = os.path.join(HERE, "fake_cudart.cpp")
LIB = os.path.join(HERE, "_build", "libfake_cudart.so")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PRELUDE = """
import ctypes, os, sys
sys.path.insert(0, %r)
fake = ctypes.CDLL(None)
fake.fake_log.restype = ctypes.c_char_p
def log():
    return [l.split() for l in fake.fake_log().decode().splitlines()]
from isosurface_gb300 import Context, IsoError, scenes
from isosurface_gb300 import source as S
""" % ROOT


def build():
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < os.path.getmtime(SRC):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        tmp = "%s.%d" % (LIB, os.getpid())
        subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", CUDA_INCLUDE, "-o", tmp, SRC])
        os.replace(tmp, LIB)
    return LIB


def run(text):
    from isosurface_gb300 import build as gbuild
    gbuild.build()
    r = subprocess.run([sys.executable, "-c", PRELUDE + text], capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, LD_PRELOAD=build()))
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
