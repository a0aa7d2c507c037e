"""Runs the library's host code on the fake runtime of fake_cudart.cpp, in a
child process (the fake is preloaded): run(script) returns what the script
printed as JSON.  The script finds `lib` (the library), `fake` (log(), clear(),
limit(bytes), used()), `ap`, `_lib`, `ctypes`, `np` and helpers for geometries
and device-pointer arguments."""
import json
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = '''
import ctypes, json, sys
import numpy as np
sys.path.insert(0, {root!r})
import apirl_b200 as ap
from apirl_b200 import _lib
from apirl_b200.geometry import ImageGeom, Sino2DGeom, Sino3DGeom
lib = _lib.load()
_g = ctypes.CDLL(None)
_g.fake_log.restype = ctypes.c_char_p
_g.fake_used.restype = ctypes.c_size_t
class fake:
    log = staticmethod(lambda: _g.fake_log().decode().splitlines())
    clear = staticmethod(lambda: _g.fake_clear())
    limit = staticmethod(lambda n: _g.fake_limit(ctypes.c_size_t(n)))
    used = staticmethod(lambda: _g.fake_used())
    launches = staticmethod(lambda: [l.split()[2] for l in fake.log() if l.startswith("launch ")])
D = ctypes.c_void_p(1 << 41)     # some device memory
S = ctypes.c_void_p(0x9990)      # some stream
def done(v):
    print("RESULT " + json.dumps(v))
'''


def build(tmp):
    so = os.path.join(str(tmp), "fake_cudart.so")
    subprocess.run(["g++", "-O1", "-fPIC", "-shared", "-std=c++17", "-I/usr/local/cuda/include",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
    return so


def run(so, script):
    env = dict(os.environ, LD_PRELOAD=so)
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT) + script], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    line = [l for l in r.stdout.splitlines() if l.startswith("RESULT ")][-1]
    return json.loads(line[7:])
