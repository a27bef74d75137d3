"""FP64 contraction of small element matrices (at most 32 entries)."""
import numpy as np
import pytest

import _synthetic as S
from sparselizard_b200 import abi
from test_gpu_split import _element_matrices, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntf,ndof,grid,norient,nterms", [
    (1, 1, 3, 1, 1), (2, 1, 9, 2, 3), (3, 3, 1, 1, 1), (3, 3, 13, 3, 2), (4, 2, 9, 1, 1), (4, 4, 4, 1, 4), (4, 4, 13, 2, 3),
    (6, 2, 9, 1, 2), (17, 1, 9, 2, 1), (5, 4, 13, 1, 2), (8, 3, 6, 2, 3), (27, 1, 9, 1, 2), (31, 1, 7, 1, 1), (8, 4, 9, 3, 2),
    (4, 4, 200, 1, 1), (3, 3, 200, 2, 1)])
def test_small_element_matrices(ctx, ntf, ndof, grid, norient, nterms):  # noqa: F811
    """Parts of 2, 4 and 8 entries, whole and cut, chunks of 32 elements, whole
    and cut, several chunks per block, several orientations, rows that are and
    are not whole sectors.  Tables and data are small whole numbers and the
    mesh, points and weights powers of two, so every sum is exact in any order
    and the element matrices equal numpy's bit for bit."""
    rng = np.random.Generator(np.random.PCG64(1000 * ntf + 10 * ndof + norient))
    gb, xyz, conn = S.group(rng, nelem_grid=grid, ntf=ntf, ndof=ndof, nterms=nterms, ngp1=2, norient=norient, ndests=1)
    g = gb.g
    x = np.arange(grid + 1.0)
    xyz = np.stack([np.tile(x, grid + 1), np.repeat(x, grid + 1), np.zeros((grid + 1) ** 2)], axis=1).ravel()
    points = np.array([[a, b] for b in (-0.5, 0.5) for a in (-0.5, 0.5)])
    np.ctypeslib.as_array(g.lagrange, (3, 4, 4))[:] = S.lagrange_q4(points)
    w = np.ctypeslib.as_array(g.weights, (4,))
    w[:] = [1.0, 0.5, 2.0, 0.25]
    E = np.ctypeslib.as_array(g.elemdata[0], (g.nelem,))
    E[:] = rng.integers(-8, 9, g.nelem)
    orient = np.ctypeslib.as_array(g.orient, (g.nelem,))
    T = []
    for k in range(g.ntables):
        t = np.ctypeslib.as_array(g.tables[k].vals, (norient, g.tables[k].rows, 4))
        t[:] = rng.integers(-4, 5, t.shape)
        T.append(t)
    ref = np.zeros((g.nelem, ntf, ndof))
    for t in range(nterms):
        g.terms[t].coef_node = 5  # the per-element coefficient alone
        M = np.einsum("oig,ojg,g->oij", T[g.terms[t].tf_table], T[g.terms[t].dof_table], w)
        ref += 0.25 * g.terms[t].scale * E[:, None, None] * M[orient]  # 0.25: the Jacobian's determinant
    got = _element_matrices(ctx, gb, xyz, conn, abi.PREC_FP64)
    assert np.array_equal(got, ref.reshape(got.shape))
