"""State that outlives a call."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import test_gpu_graphs as T
from sparselizard_b200 import abi

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _compile(tmp_path, name, code):
    src, lib = tmp_path / f"{name}.cpp", tmp_path / f"{name}.so"
    src.write_text(code)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "sparselizard_b200", "csrc"), "-I", "/usr/local/cuda/include", str(src), "-o", str(lib), "-ldl"],
                   check=True)
    return str(lib)


def test_timeout_flag_of_an_earlier_call(tmp_path):
    """The time-out flag left set by a call that ended before reading it (set
    here through the context's own pointer) belongs to that call: the next
    steps, in FP64 and in split precision, return their values."""
    peek = ctypes.CDLL(_compile(tmp_path, "peek", """
#include "engine_internal.h"
extern "C" unsigned int* flag(void* ctx) { return static_cast<slgpu::Ctx*>(ctx)->main.split_flag; }
"""))
    peek.flag.restype, peek.flag.argtypes = ctypes.POINTER(ctypes.c_uint), [ctypes.c_void_p]
    ctx = abi.Context(0)
    t = T._setup(ctx, np.random.Generator(np.random.PCG64(52)), 0, 20, 9, 9, 2, 2, 600)
    ref = {p: T._process(ctx, t, p) for p in (abi.PREC_SPLIT, abi.PREC_FP64)}
    flag = peek.flag(ctx.h)
    for p in (abi.PREC_FP64, abi.PREC_SPLIT, abi.PREC_SPLIT, abi.PREC_SPLIT):  # at last replayed from a graph
        flag[0] = 1
        A, D = T._process(ctx, t, p)
        assert flag[0] == 0 and np.array_equal(A, ref[p][0]) and np.array_equal(D, ref[p][1])
    ctx.close()
