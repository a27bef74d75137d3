"""Matrices of many groups, beyond what one launch takes, and patterns with raw fragments in long rows."""
import ctypes
import os
import sys

import numpy as np
import pytest

import _synthetic as S
from sparselizard_b200 import abi

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import slref  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = abi.Context(0)
    yield c
    c.close()


def _matrix(ctx, groups, xyz, conn, ndofs, frags=()):
    L = ctx.lib
    ctx.check(L.slgpu_mesh_set_nodes(ctx.h, 0, xyz.size // 3, abi.f64p(xyz)))
    ctx.check(L.slgpu_mesh_set_elements(ctx.h, 0, 3, 4, conn.size // 4, abi.i32p(conn)))
    h = ctypes.c_int()
    ctx.check(L.slgpu_matrix_create(ctx.h, ndofs, ctypes.byref(h)))
    for g in groups:
        ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g), None))
    for ntr, ndr, nr, nc, rows, cols, vals in frags:
        ctx.check(L.slgpu_matrix_add_fragment(ctx.h, h, ntr, ndr, nr, nc, abi.i32p(rows), abi.i32p(cols), abi.f64p(vals)))
    return h.value


def _check(ctx, h, con, precision, ref, mag, tol):
    L, info = ctx.lib, abi.CsrInfo()
    ctx.check(L.slgpu_matrix_process(ctx.h, h, con.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), precision, ctypes.byref(info)))
    out = {k: np.zeros(max(1, n), t) for k, n, t in (("Arows", info.nA + 1, np.int32), ("Acols", info.nnzA, np.int32),
                                                     ("Avals", info.nnzA, np.float64), ("Drows", info.nA + 1, np.int32),
                                                     ("Dcols", info.nnzD, np.int32), ("Dvals", info.nnzD, np.float64))}
    ctx.check(L.slgpu_matrix_download(ctx.h, h, *[abi.i32p(v) if v.dtype == np.int32 else abi.f64p(v) for v in out.values()]))
    for k in ("Arows", "Acols", "Drows", "Dcols"):
        assert np.array_equal(out[k][: ref[k].size], ref[k]), f"{k} differs"
    for k in ("Avals", "Dvals"):
        err = np.abs(out[k][: ref[k].size] - ref[k]) / np.maximum(mag[k], 1e-300)
        assert not err.size or err.max() <= tol, f"{k}: {err.max():.3e}"


def _launches(ctx, family):
    ms, n, w = ctypes.c_double(), ctypes.c_int64(), ctypes.c_double()
    ctx.check(ctx.lib.slgpu_kernel_stats(ctx.h, family.encode(), ctypes.byref(ms), ctypes.byref(n), ctypes.byref(w)))
    return n.value


@pytest.mark.parametrize("ngp1", [2, 3, 7])
def test_many_groups(ctx, ngp1):
    """36 groups of one geometry with different shapes and numbers of terms:
    30 go through the split kernels (24 to a launch; their slices 16 groups to
    a kernel, several rounds of groups to a block), 6, among them the first,
    have small element matrices.  Against the oracle, and by the number of
    launches of each family: the coefficients of split groups stay out of
    memory."""
    shapes = [(4, 4, 2), (8, 8, 2), (9, 9, 3), (10, 8, 1), (12, 9, 4), (8, 11, 2)]
    built = [S.group(np.random.Generator(np.random.PCG64(70)), nelem_grid=9, ntf=ntf, ndof=ndof, nterms=nt, ngp1=ngp1, norient=2,
                     ndests=1 + k % 2, ndofs=300 + k) for k, (ntf, ndof, nt) in enumerate(shapes * 6)]
    groups, (_, xyz, conn) = [b[0].g for b in built], built[0]
    ndofs = 340
    con = (np.random.Generator(np.random.PCG64(71)).random(ndofs) < 0.1).astype(np.uint8)
    conns = [conn] * len(groups)
    ref = slref.matrix(groups, xyz, conns, ndofs, con)
    mag = slref.matrix(groups, xyz, conns, ndofs, con, absmode=True)
    h = _matrix(ctx, groups, xyz, conn, ndofs)
    for prec, tol in ((abi.PREC_FP64, 1e-12), (abi.PREC_SPLIT, 1e-10), (abi.PREC_FP32, 1e-6)):
        for _ in range(3):  # tuned, plain, captured
            _check(ctx, h, con, prec, ref, mag, tol)
        split = {abi.PREC_SPLIT: "contract_split", abi.PREC_FP32: "contract_split_fp32"}.get(prec)
        assert _launches(ctx, "coefficients") == 1
        assert _launches(ctx, "slice_cols") == (2 if split else 0)
        if split:
            assert _launches(ctx, split) == 2
        assert _launches(ctx, "contract_fp64") >= (6 if split else 8)
    ctx.check(ctx.lib.slgpu_matrix_destroy(ctx.h, h))


@pytest.mark.parametrize("length", [1, 700, 5400, 5500])
def test_pattern_with_fragments(ctx, length):
    """A raw fragment that gives row 3 `length` more COO entries (columns
    repeated, some dropped) and one of several rows and columns, beside a
    group: on both sides of the longest row that is built by itself.  CSR
    structure equal to the oracle's, values within 1e-12 of the sums of
    magnitudes."""
    rng = np.random.Generator(np.random.PCG64(72 + length))
    ndofs = 4000
    gb, xyz, conn = S.group(rng, nelem_grid=8, ntf=3, ndof=4, nterms=2, ngp1=2, norient=1, ndests=1, ndofs=ndofs)
    frags = [(1, length, length, 1, np.array([3], np.int32), rng.integers(-1, ndofs, length).astype(np.int32), rng.standard_normal(length)),
             (3, 2, 6, 5, rng.integers(-1, ndofs, 15).astype(np.int32), rng.integers(-1, ndofs, 10).astype(np.int32), rng.standard_normal(30))]
    con = (rng.random(ndofs) < 0.1).astype(np.uint8)
    con[3] = 0
    ref = slref.matrix([gb.g], xyz, [conn], ndofs, con, frags)
    mag = slref.matrix([gb.g], xyz, [conn], ndofs, con, frags, absmode=True)
    h = _matrix(ctx, [gb.g], xyz, conn, ndofs, frags)
    _check(ctx, h, con, abi.PREC_FP64, ref, mag, 1e-12)
    ctx.check(ctx.lib.slgpu_matrix_destroy(ctx.h, h))
