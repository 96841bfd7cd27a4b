"""The library's host side over tests/native/runtime_stub.cpp: `run(script)`
links the library's objects with it and runs a Python script in a process of its
own, with `A` (apogee_gpu over that library), `C` (circuits), `stub` (its extra
functions) and `addr(data)` (the "device" address of some bytes) at hand. What the
script leaves in `result` comes back."""
import glob
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "apogee-vm_gb300")

PRELUDE = """
import ctypes, json, os, random, sys, time
import apogee_gpu as A
import circuits as C
_lib = A.lib()
class stub:
    @staticmethod
    def _text(f):
        f.restype = ctypes.c_size_t
        buf = ctypes.create_string_buffer(1 << 16)
        f(buf, ctypes.c_size_t(len(buf)))
        return [line for line in buf.value.decode().split("\\n") if line]
    @staticmethod
    def misplaced():
        return stub._text(_lib.stub_misplaced)
    @staticmethod
    def launched():
        return {line.rsplit(" ", 1)[0]: int(line.rsplit(" ", 1)[1]) for line in stub._text(_lib.stub_launched)}
    @staticmethod
    def reset():
        _lib.stub_reset()
    @staticmethod
    def most():
        _lib.stub_most.restype = ctypes.c_size_t
        return _lib.stub_most()
    @staticmethod
    def held():
        _lib.stub_held.restype = ctypes.c_size_t
        return _lib.stub_held()
_kept = []
def addr(data):
    # 256-byte aligned, as device memory is
    buf = ctypes.create_string_buffer(len(data) + 256)
    a = ctypes.addressof(buf)
    a += -a % 256
    ctypes.memmove(a, bytes(data), len(data))
    _kept.append(buf)
    return a
result = None
"""


def library() -> str:
    sys.path.insert(0, PKG)
    import build_lib

    build_lib.build()
    out = os.path.join(build_lib.BUILD, "libapogee_stub.so")
    src = os.path.join(ROOT, "tests", "native", "runtime_stub.cpp")
    objs = sorted(glob.glob(os.path.join(build_lib.BUILD, "*.o")))
    if build_lib._stale(out, objs + [src]):
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        tmp = f"{out}.{os.getpid()}"
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(cuda, "include"), src]
                              + objs + ["-o", tmp, "-lpthread"])
        os.replace(tmp, out)
    return out


def run(script: str, timeout: float = 300):
    env = dict(os.environ, APOGEE_GPU_LIB=library(), PYTHONPATH=os.pathsep.join([PKG, os.path.join(ROOT, "tests")]))
    p = subprocess.run([sys.executable, "-c", PRELUDE + script + "\nprint('RESULT ' + json.dumps(result))"], env=env,
                       capture_output=True, text=True, timeout=timeout)
    assert p.returncode == 0, p.stderr[-4000:]
    return json.loads(p.stdout.rsplit("RESULT ", 1)[1])
