"""Runs scripts against the library linked with a CUDA runtime that needs no
GPU (tests/cpp/fake_cuda.cpp): tests of its host code, of which kernels a call
launches, and of failures that no GPU is to be brought to."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = """
import ctypes, os, subprocess
from pathlib import Path
from qflex_gb300 import _lib
_lib.LIB_PATH = Path(os.environ["QFLEX_FAKE_LIB"])
from qflex_gb300 import *
from qflex_gb300 import rqc
fake = _lib.load_library()
fake.fake_log.restype = ctypes.c_char_p
fake.fake_memory.argtypes = fake.fake_largest_block.argtypes = [ctypes.c_size_t]
fake.fake_capturing.argtypes = [ctypes.c_void_p, ctypes.c_int]
def log():
    "The runtime's calls since the last time, without stream and event creation."
    text = fake.fake_log().decode()
    fake.fake_clear()
    return text.splitlines()
def kernels(lines=None):
    "The kernels of the launches in the log: name<template arguments>."
    names = [x.split()[-1] for x in (log() if lines is None else lines) if x.startswith("launch")]
    text = subprocess.run(["c++filt", "-p"], input="\\n".join(names), capture_output=True, text=True, check=True).stdout
    return [x.split("::")[-1] for x in text.splitlines() if x]
A, B, C = 1 << 40, 1 << 41, 1 << 42  # addresses: no kernel runs
"""


@pytest.fixture(scope="session")
def fake_lib(built_lib, tmp_path_factory):
    """The library's object files with the fake runtime."""
    out = tmp_path_factory.mktemp("fake_cuda") / "libqflex_gb300.so"
    objects = sorted(str(o) for o in (ROOT / "qflex_gb300" / "_build").glob("*.o")
                     if (ROOT / "qflex_gb300" / "csrc" / o.stem).exists())
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++20", "-I", "/usr/local/cuda/include",
                    str(ROOT / "tests" / "cpp" / "fake_cuda.cpp"), *objects, "-o", str(out), "-lpthread"], check=True)
    return out


@pytest.fixture
def run_fake(fake_lib):
    """Runs a script in a process of its own; its standard output."""
    def run(script, **env):
        r = subprocess.run([sys.executable, "-c", PRELUDE + script], cwd=ROOT, capture_output=True, text=True,
                           env={**os.environ, "QFLEX_FAKE_LIB": str(fake_lib), **env}, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return run
