"""Split precision on operands of few significant bits, on quotients that are exact, and at the ends of the range."""
import os
import subprocess
import sys

import numpy as np
import pytest

import _synthetic as S
from sparselizard_b200 import abi
from test_gpu_split import _element_matrices

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def whole_numbers(seed, ntf, ndof, nterms, norient, grid, coef, size=(1.0, 1.0), elem=1000):
    """A group on rectangles of the given size whose tables and data are whole
    numbers and whose points and weights are powers of two, with the
    coefficient node `coef` (5: the element data; 6: entry (0, 0) of the
    inverse Jacobian, 2 / size[0]), and its element matrices: exact sums."""
    rng = np.random.Generator(np.random.PCG64(seed))
    gb, xyz, conn = S.group(rng, nelem_grid=grid, ntf=ntf, ndof=ndof, nterms=nterms, ngp1=2, norient=norient, ndests=1)
    g = gb.g
    x = np.arange(grid + 1.0)
    xyz = np.stack([size[0] * np.tile(x, grid + 1), size[1] * np.repeat(x, grid + 1), np.zeros((grid + 1) ** 2)], axis=1).ravel()
    points = np.array([[a, b] for b in (-0.5, 0.5) for a in (-0.5, 0.5)])
    np.ctypeslib.as_array(g.lagrange, (3, 4, 4))[:] = S.lagrange_q4(points)
    w = np.ctypeslib.as_array(g.weights, (4,))
    w[:] = [1.0, 0.5, 2.0, 0.25]
    E = np.ctypeslib.as_array(g.elemdata[0], (g.nelem,))
    E[:] = rng.integers(-elem, elem + 1, g.nelem)
    orient = np.ctypeslib.as_array(g.orient, (g.nelem,))
    T = []
    for k in range(g.ntables):
        t = np.ctypeslib.as_array(g.tables[k].vals, (norient, g.tables[k].rows, 4))
        t[:] = rng.integers(-100, 101, t.shape)
        T.append(t)
    ref = np.zeros((g.nelem, ntf, ndof))
    c = E if coef == 5 else np.full(g.nelem, 2.0 / size[0])
    for t in range(nterms):
        g.terms[t].coef_node = coef
        M = np.einsum("oig,ojg,g->oij", T[g.terms[t].tf_table], T[g.terms[t].dof_table], w)
        ref += 0.25 * size[0] * size[1] * g.terms[t].scale * c[:, None, None] * M[orient]
    return gb, xyz, conn, ref.reshape(g.nelem, ntf * ndof)


def check_whole(ctx, **kw):
    gb, xyz, conn, ref = whole_numbers(**kw)
    assert np.abs(ref).max() > 0
    for prec in (abi.PREC_FP64, abi.PREC_SPLIT, abi.PREC_FP32):
        got = _element_matrices(ctx, gb, xyz, conn, prec)
        want = ref.astype(np.float32).astype(np.float64) if prec == abi.PREC_FP32 else ref
        assert np.array_equal(got, want), f"precision {prec}: {np.abs(got - want).max()} of {np.abs(want).max()}"


def check_whole_all():
    ctx = abi.Context(0)
    for k, (ntf, ndof, nterms, norient, grid) in enumerate([(9, 9, 1, 1, 9), (9, 9, 3, 2, 13), (27, 27, 4, 1, 20), (10, 8, 9, 3, 7)]):
        check_whole(ctx, seed=70 + k, ntf=ntf, ndof=ndof, nterms=nterms, norient=norient, grid=grid, coef=5)
    ctx.close()


@pytest.mark.parametrize("interpreter", ["0", "1"])
def test_whole_numbers_are_exact(interpreter):
    """Tables and coefficients of at most 21 significant bits: every product
    and sum is exact, so the element matrices of each tier equal numpy's bit for
    bit (rounded to floats in the FP32-level tier), whether the coefficients go
    straight to slices or through memory."""
    env = dict(os.environ, SLGPU_COEF_INTERPRETER=interpreter, PYTHONPATH=os.pathsep.join([HERE, os.path.dirname(HERE)]))
    subprocess.run([sys.executable, "-c", "import test_gpu_exact as T; T.check_whole_all()"], env=env, check=True, timeout=300)


@pytest.mark.parametrize("size", [(2.0, 98.0), (2.0, 206.0)])
def test_inverse_jacobian_is_divided(size):
    """Cofactors are divided by the determinant: 49 / 49 and 103 / 103 are 1
    (times the rounded reciprocal, they are not), so the element matrices are
    whole numbers, exact in each tier."""
    ctx = abi.Context(0)
    check_whole(ctx, seed=80, ntf=9, ndof=9, nterms=2, norient=1, grid=9, coef=6, size=size)
    ctx.close()


@pytest.mark.parametrize("largest,table", [(1.79e308, 1e-10), (1e308, 1e-10), (3e-315, 1.0)])
def test_ends_of_the_range(largest, table):
    """Coefficients up to the largest double, and ones of which none is a
    normal double: within 1e-10 of FP64's element matrices; a zero column
    stays zero."""
    ctx = abi.Context(0)
    gb, xyz, conn, _ = whole_numbers(seed=90, ntf=9, ndof=9, nterms=1, norient=1, grid=13, coef=5)
    g = gb.g
    g.terms[0].scale = 1.0
    np.ctypeslib.as_array(g.weights, (4,))[:] = [4.0, 2.0, 1.0, 0.5]  # times the determinant 1/4
    np.ctypeslib.as_array(g.tables[0].vals, (1, 9, 4))[:] *= table
    e = np.ctypeslib.as_array(g.elemdata[0], (g.nelem,))
    e[:] = largest * np.random.Generator(np.random.PCG64(91)).uniform(0.3, 1.0, g.nelem)
    e[0], e[5] = largest, 0.0
    ref = _element_matrices(ctx, gb, xyz, conn, abi.PREC_FP64)
    got = _element_matrices(ctx, gb, xyz, conn, abi.PREC_SPLIT)
    assert np.isfinite(ref).all() and np.isfinite(got).all() and not got[5].any()
    size = np.abs(ref).max(axis=1)
    assert (size > 0).sum() == g.nelem - 1
    assert (np.abs(got - ref).max(axis=1) <= 1e-10 * size).all()
    ctx.close()
