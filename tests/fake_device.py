"""Runs a script against libgw.so over tests/fake_cudart.cpp, in a process of its own."""
import os
import subprocess
import sys
import textwrap
from pathlib import Path

from gundam_gb300 import build as B

HERE = Path(__file__).resolve().parent

PRELUDE = """
import ctypes, sys
sys.path.insert(0, {root!r})
import numpy as np
from gundam_gb300 import Engine, Workload
from gundam_gb300 import _native as N
from gundam_gb300.surrogate import MLP, Surrogate

_fake = ctypes.CDLL({fake!r})
def log():
    b = ctypes.create_string_buffer(1 << 20)
    _fake.fake_take(b, ctypes.c_size_t(len(b)))
    return b.value.decode().splitlines()
"""


def run(script: str, tmp_path) -> None:
    """Runs `script` after PRELUDE; its assertions are the caller's."""
    fake = tmp_path / "libfake_cudart.so"
    include = Path(B._nvcc()).resolve().parent.parent / "include"
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-fPIC", "-shared", "-pthread", "-I",
                    str(include), str(HERE / "fake_cudart.cpp"), "-o", str(fake)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(fake))
    code = PRELUDE.format(root=str(HERE.parent), fake=str(fake)) + textwrap.dedent(script)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-4000:]
