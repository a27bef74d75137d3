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


def test_shared_memory_limits_per_context(tmp_path):
    """Two contexts in one process (on two devices, in a program with two):
    each raises the dynamic shared-memory limit of every kernel that it
    launches beyond the default, since the limit belongs to the device.  The
    calls are counted by a library loaded before the CUDA runtime."""
    shim = _compile(tmp_path, "count", """
#include <dlfcn.h>
#include <map>
static std::map<const void*, int> calls;
extern "C" int cudaFuncSetAttribute(const void* f, int attr, int value)
{
    static auto real = reinterpret_cast<int (*)(const void*, int, int)>(dlsym(dlopen("libcudart.so.12", RTLD_NOW), "cudaFuncSetAttribute"));
    calls[f]++;
    return real(f, attr, value);
}
extern "C" int functions() { return (int)calls.size(); }
extern "C" int fewest() { int n = 1 << 30; for (auto& c : calls) n = c.second < n ? c.second : n; return n; }
""")
    code = """
import ctypes
import numpy as np
from sparselizard_b200 import abi
import test_gpu_graphs as T
shim = ctypes.CDLL(None)
seen = []
for k in range(2):
    ctx = abi.Context(0)
    for ntf, ndof, ndofs in ((4, 4, 3000), (9, 9, 60), (8, 8, 9000), (40, 40, 7000)):  # many entries per row, and rows of many columns
        t = T._setup(ctx, np.random.Generator(np.random.PCG64(53)), 0, 40, ntf, ndof, 2, 2, ndofs)
        for p in (abi.PREC_FP64, abi.PREC_SPLIT, abi.PREC_FP32):
            T._process(ctx, t, p)
    ctx.close()
    seen.append(shim.functions())
assert seen[0] >= 5 and seen[0] == seen[1], seen
assert shim.fewest() >= 2, "a kernel's limit was not raised again in the second context"
"""
    env = dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=os.pathsep.join([HERE, ROOT]))
    subprocess.run([sys.executable, "-c", code], env=env, check=True, timeout=300)


def test_server_arena_holds_what_requests_use():
    """What preparing a template reserves for split-precision requests: the
    element matrices, the values and the replaced data (an eighth more, for
    the arena grows so), and the slices and their scales; not the
    coefficients, which are never in memory.  A request then adds nothing."""
    import test_gpu_serving as V
    from sparselizard_b200 import serving

    ctx = abi.Context(0)
    rng = np.random.Generator(np.random.PCG64(54))
    t = V._template(ctx, rng, 1, 150, 9, 9, 9, 4, 2500)
    g, n = t["gb"].g, t["nmesh"]
    srv = serving.Server(ctx.lib, ctx.h, 1)
    b0 = ctx.lib.slgpu_bytes_in_use(ctx.h)
    srv.prepare(t["handle"], abi.PREC_SPLIT)
    b1 = ctx.lib.slgpu_bytes_in_use(ctx.h)
    tiles = n // 64 + 2  # of each of two orientations
    slices = 6 * (9 * 16 + 16) // 32 * 32 * tiles * 64 + 8 * 64 * tiles
    rows = 2 * 7 * 128 * 160 + (1 << 20)  # row slices and small tables
    arena = 8 * (81 * n + t["nnzA"] + t["nnzD"] + 2 * n) + (1 << 20)
    assert b1 - b0 <= 9 * arena // 8 + slices + rows, f"{b1 - b0} bytes reserved"
    A, D = np.zeros(t["nnzA"]), np.zeros(t["nnzD"])
    up = serving.UpdateSpec(0, abi.UPDATE_ELEMDATA, 0, rng.lognormal(0.0, 0.4, n))
    assert srv.wait(srv.submit(t["handle"], abi.PREC_SPLIT, [up], A, D)).status == abi.OK
    assert ctx.lib.slgpu_bytes_in_use(ctx.h) <= b1
    srv.close()
    ctx.close()
