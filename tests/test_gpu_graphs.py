"""CUDA-graph replay of process() on a resident pattern.

The value path (coefficients, contractions, CSR values) of a matrix is
captured into a graph on the second process() with unchanged launches and
replayed afterwards.  Replays must give the same values bit for bit as the
ungraphed path, also after in-place changes of per-element data, node
coordinates, term scales and destination multipliers (read by the kernels at
run time).  Both CSR value kernels (streaming warps, warp per row) must agree
bit for bit as well.
"""
import ctypes

import numpy as np
import pytest

import _synthetic as S
from sparselizard_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = abi.Context(0)
    yield c
    c.close()


def _setup(ctx, rng, mesh_id, grid, ntf, ndof, nterms, ngp1, ndofs):
    gb, xyz, conn = S.group(rng, nelem_grid=grid, ntf=ntf, ndof=ndof, nterms=nterms, ngp1=ngp1, norient=2, ndests=2,
                            ndofs=ndofs)
    g = gb.g
    g.mesh = mesh_id
    L = ctx.lib
    ctx.check(L.slgpu_mesh_set_nodes(ctx.h, mesh_id, xyz.size // 3, abi.f64p(xyz)))
    ctx.check(L.slgpu_mesh_set_elements(ctx.h, mesh_id, 3, 4, conn.size // 4, abi.i32p(conn)))
    h = ctypes.c_int()
    ctx.check(L.slgpu_matrix_create(ctx.h, ndofs, ctypes.byref(h)))
    ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g), None))
    con = (rng.random(ndofs) < 0.1).astype(np.uint8)
    return dict(gb=gb, h=h.value, con=con, xyz=xyz, nelem=g.nelem, nterms=g.nterms, ndests=g.ndests, mesh=mesh_id)


def _process(ctx, t, precision):
    L = ctx.lib
    info = abi.CsrInfo()
    ctx.check(L.slgpu_matrix_process(ctx.h, t["h"], t["con"].ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), precision,
                                     ctypes.byref(info)))
    A, D = np.zeros(max(1, info.nnzA)), np.zeros(max(1, info.nnzD))
    ctx.check(L.slgpu_matrix_download_values(ctx.h, t["h"], abi.f64p(A), abi.f64p(D)))
    return A[: info.nnzA].copy(), D[: info.nnzD].copy()


def _run(ctx, t, precision, graphs, edits):
    """process() after each edit (a callable or None); returns the values."""
    ctx.check(ctx.lib.slgpu_ctx_set_graphs(ctx.h, 1 if graphs else 0))
    out = []
    for e in edits:
        if e is not None:
            e()
        out.append(_process(ctx, t, precision))
    return out


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_SPLIT])
def test_graph_replay_matches_ungraphed(ctx, precision):
    rng = np.random.Generator(np.random.PCG64(21))
    t = _setup(ctx, rng, 11 + precision, 60, 9, 9, 4, 3, 3000)
    L = ctx.lib
    e1 = rng.lognormal(0.0, 0.4, t["nelem"])
    e2 = rng.lognormal(0.0, 0.4, t["nelem"])
    xyz2 = t["xyz"] * 1.01
    scales = rng.uniform(0.5, 2.0, t["nterms"])
    mults = rng.uniform(-2.0, 2.0, t["ndests"])

    def set_e(v):
        return lambda: ctx.check(L.slgpu_matrix_set_elemdata(ctx.h, t["h"], 0, 0, abi.f64p(v)))

    def set_nodes(v):
        return lambda: ctx.check(L.slgpu_mesh_set_nodes(ctx.h, t["mesh"], v.size // 3, abi.f64p(v)))

    def set_scales(ts, dm):
        return lambda: ctx.check(L.slgpu_matrix_set_scales(ctx.h, t["h"], 0, abi.f64p(ts) if ts is not None else None,
                                                           abi.f64p(dm) if dm is not None else None))

    orig_scales = np.zeros(t["nterms"])
    orig_mults = np.zeros(t["ndests"])
    ctx.check(L.slgpu_matrix_get_scales(ctx.h, t["h"], 0, abi.f64p(orig_scales), abi.f64p(orig_mults)))
    edits = [set_e(e1), None, None, set_e(e2), set_nodes(xyz2), set_scales(scales, None), None,
             set_scales(None, mults), None, set_nodes(t["xyz"]), set_scales(orig_scales, orig_mults)]
    g0 = L.slgpu_graph_launches(ctx.h)
    with_graph = _run(ctx, t, precision, True, edits)
    replays = L.slgpu_graph_launches(ctx.h) - g0
    without = _run(ctx, t, precision, False, edits)
    ctx.check(L.slgpu_ctx_set_graphs(ctx.h, 1))
    assert replays >= 8, f"only {replays} graph replays"
    for i, ((a, d), (a0, d0)) in enumerate(zip(with_graph, without)):
        assert np.all(np.isfinite(a)) and np.all(np.isfinite(d)), f"call {i}: non-finite values"
        assert np.array_equal(a, a0) and np.array_equal(d, d0), f"call {i}: graph != ungraphed"
    # The edits changed the values (the replays are not stale copies).
    assert not np.array_equal(with_graph[2][0], with_graph[3][0])
    assert not np.array_equal(with_graph[3][0], with_graph[4][0])
    assert not np.array_equal(with_graph[6][0], with_graph[7][0])


def test_graph_kernel_stats_and_launch_count(ctx):
    rng = np.random.Generator(np.random.PCG64(22))
    t = _setup(ctx, rng, 13, 40, 4, 4, 3, 2, 1200)
    L = ctx.lib
    ctx.check(L.slgpu_ctx_set_graphs(ctx.h, 1))
    for _ in range(3):
        _process(ctx, t, abi.PREC_FP64)
    k0 = L.slgpu_kernel_launches(ctx.h)
    g0 = L.slgpu_graph_launches(ctx.h)
    _process(ctx, t, abi.PREC_FP64)
    assert L.slgpu_graph_launches(ctx.h) == g0 + 1
    # coefficients, contraction, CSR values
    assert L.slgpu_kernel_launches(ctx.h) - k0 == 3
    ms, n, w = ctypes.c_double(), ctypes.c_int64(), ctypes.c_double()
    for fam in ("coefficients", "contract_fp64", "row_values"):
        ctx.check(L.slgpu_kernel_stats(ctx.h, fam.encode(), ctypes.byref(ms), ctypes.byref(n), ctypes.byref(w)))
        assert n.value == 1 and ms.value > 0 and w.value > 0, fam


def test_value_kernels_agree(tmp_path):
    """The streaming-warp, warp-per-row and thread-per-row CSR value kernels,
    each forced in a child process, give the same values bit for bit
    (incidence widths 4, 9 and 40; the thread kernel on the short rows)."""
    import os
    import subprocess
    import sys

    here = os.path.dirname(os.path.abspath(__file__))
    res = {}
    for k in ("stream", "warp", "thread"):
        out = str(tmp_path / f"{k}.npz")
        env = dict(os.environ, SLGPU_ROW_KERNEL=k)
        subprocess.run([sys.executable, os.path.join(here, "_rowkernel_child.py"), out], env=env, check=True, timeout=600)
        res[k] = np.load(out)
    for key in res["warp"].files:
        for k in ("stream", "thread"):
            a, b = res[k][key], res["warp"][key]
            assert np.all(np.isfinite(a)), key
            assert np.array_equal(a, b), f"{key}: {k} and warp-per-row value kernels differ"


@pytest.mark.parametrize("grid,ndofs,mult,dup", [(60, 3000, 1.0, False), (200, 30000, 3.0, True), (400, 150000, 1.0, True),
                                                 (400, 150000, -2.5, False), (600, 1200000, 1.0, False)])
def test_rows_of_a_warp(tmp_path, grid, ndofs, mult, dup):
    """1 to 31 rows per warp, rows of one to thousands of incidences that start
    and end anywhere in a window of 32, with and without serial incidences and
    multipliers: the warp kernel's values equal the streaming kernel's bit for
    bit (each forced in its own process)."""
    import os
    import subprocess
    import sys

    code = """
import ctypes, sys
import numpy as np
import _synthetic as S
from sparselizard_b200 import abi
rng = np.random.Generator(np.random.PCG64(41))
grid, ndofs, mult, dup = %d, %d, %r, %r
gb, xyz, conn = S.group(rng, nelem_grid=grid, ntf=4, ndof=4, nterms=1, ngp1=2, norient=1, ndests=1, ndofs=ndofs)
g = gb.g
g.dests[0].multiplier = mult
t = np.ctypeslib.as_array(g.dests[0].tfaddr, (4, g.nelem))
d = np.ctypeslib.as_array(g.dests[0].dofaddr, (4, g.nelem))
d[:] = (t[::-1] // 16 * 16 + rng.integers(0, 16, d.shape)) %% ndofs  # rows stay short
t[:, ::97] = rng.integers(0, 40, t[:, ::97].shape)  # and some have many incidences
if dup:
    d[1, ::13] = d[0, ::13]
ctx = abi.Context(0)
L = ctx.lib
ctx.check(L.slgpu_mesh_set_nodes(ctx.h, 0, xyz.size // 3, abi.f64p(xyz)))
ctx.check(L.slgpu_mesh_set_elements(ctx.h, 0, 3, 4, conn.size // 4, abi.i32p(conn)))
h = ctypes.c_int()
ctx.check(L.slgpu_matrix_create(ctx.h, ndofs, ctypes.byref(h)))
ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g), None))
con = (rng.random(ndofs) < 0.05).astype(np.uint8)
info = abi.CsrInfo()
ctx.check(L.slgpu_matrix_process(ctx.h, h, con.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), abi.PREC_FP64, ctypes.byref(info)))
A, D = np.zeros(max(1, info.nnzA)), np.zeros(max(1, info.nnzD))
ctx.check(L.slgpu_matrix_download_values(ctx.h, h, abi.f64p(A), abi.f64p(D)))
np.savez(sys.argv[1], A=A, D=D)
""" % (grid, ndofs, mult, dup)
    here = os.path.dirname(os.path.abspath(__file__))
    res = {}
    for k in ("stream", "warp"):
        out = str(tmp_path / f"{k}.npz")
        env = dict(os.environ, SLGPU_ROW_KERNEL=k, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
        subprocess.run([sys.executable, "-c", code, out], env=env, check=True, timeout=300)
        res[k] = np.load(out)
    for key in ("A", "D"):
        assert np.all(np.isfinite(res["warp"][key])) and np.abs(res["warp"][key]).max() > 0
        assert np.array_equal(res["warp"][key], res["stream"][key]), key


def test_graph_replay_with_transposed_pair(ctx):
    """A matrix with two transposed-partner groups, edited so that the pairing
    turns off and on again (a scale of one group; element data of one group,
    then of both): replayed graphs give the ungraphed values bit for bit, and
    the pairing follows the edits."""
    rng = np.random.Generator(np.random.PCG64(23))
    ndofs = 2500
    gb, xyz, conn = S.group(rng, nelem_grid=40, ntf=12, ndof=8, nterms=4, ngp1=3, norient=2, ndests=1, ndofs=ndofs)
    g1 = gb.g
    g2 = abi.Group.from_buffer_copy(g1)
    g2.ntf, g2.ndof = g1.ndof, g1.ntf
    terms2 = (abi.Term * g1.nterms)(*[abi.Term(g1.terms[t].dof_table, g1.terms[t].tf_table, g1.terms[t].coef_node, 0,
                                               g1.terms[t].scale) for t in range(g1.nterms)])
    g2.terms = terms2
    dest2 = (abi.Dest * 1)()
    dest2[0].tfaddr, dest2[0].dofaddr, dest2[0].multiplier = g1.dests[0].dofaddr, g1.dests[0].tfaddr, 1.5
    g2.dests = dest2
    mesh_id = 31
    g1.mesh = g2.mesh = mesh_id
    L = ctx.lib
    ctx.check(L.slgpu_mesh_set_nodes(ctx.h, mesh_id, xyz.size // 3, abi.f64p(xyz)))
    ctx.check(L.slgpu_mesh_set_elements(ctx.h, mesh_id, 3, 4, conn.size // 4, abi.i32p(conn)))
    h = ctypes.c_int()
    ctx.check(L.slgpu_matrix_create(ctx.h, ndofs, ctypes.byref(h)))
    ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g1), None))
    ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g2), None))
    t = dict(h=h.value, con=(rng.random(ndofs) < 0.1).astype(np.uint8))
    sc = np.zeros(g1.nterms)
    ctx.check(L.slgpu_matrix_get_scales(ctx.h, t["h"], 0, abi.f64p(sc), None))
    sc2 = sc.copy()
    sc2[1] *= 3.0
    e_old = np.ctypeslib.as_array(g1.elemdata[0], (g1.nelem,)).copy()
    e_new = rng.lognormal(0.0, 0.4, g1.nelem)

    def set_scales(gi, v):
        return lambda: ctx.check(L.slgpu_matrix_set_scales(ctx.h, t["h"], gi, abi.f64p(v), None))

    def set_e(gi, v):
        return lambda: ctx.check(L.slgpu_matrix_set_elemdata(ctx.h, t["h"], gi, 0, abi.f64p(v)))

    def partner():
        pt = ctypes.c_int32()
        ctx.check(L.slgpu_matrix_group_symmetry(ctx.h, t["h"], 0, None, None, ctypes.byref(pt)))
        return pt.value

    edits = [None, None, set_scales(0, sc2), None, None, set_scales(1, sc2), None, None, set_e(1, e_new), None,
             set_e(0, e_new), None, None, set_e(0, e_old), set_e(1, e_old), set_scales(0, sc), set_scales(1, sc), None]
    paired = [True, True, False, False, False, True, True, True, False, False, True, True, True, False, True, False, True,
              True]

    def run(graphs):
        ctx.check(L.slgpu_ctx_set_graphs(ctx.h, 1 if graphs else 0))
        out = []
        for e, p in zip(edits, paired):
            if e is not None:
                e()
            assert (partner() == 1) == p
            out.append(_process(ctx, t, abi.PREC_SPLIT))
        return out

    g0 = L.slgpu_graph_launches(ctx.h)
    with_graph = run(True)
    replays = L.slgpu_graph_launches(ctx.h) - g0
    without = run(False)
    ctx.check(L.slgpu_ctx_set_graphs(ctx.h, 1))
    ctx.check(L.slgpu_matrix_destroy(ctx.h, t["h"]))
    assert replays >= 5, f"only {replays} graph replays"
    for i, ((a, d), (a0, d0)) in enumerate(zip(with_graph, without)):
        assert np.all(np.isfinite(a)) and np.all(np.isfinite(d)), f"call {i}: non-finite values"
        assert np.array_equal(a, a0) and np.array_equal(d, d0), f"call {i}: graph != ungraphed"
    assert not np.array_equal(with_graph[1][0], with_graph[2][0])


def test_pattern_serial_and_page_locked_downloads(ctx):
    """slgpu_matrix_pattern_serial: unchanged across process() calls on the same
    addresses and constraints, new when the constraints change.  Values
    downloaded into page-locked host memory (slgpu_host_register) equal those
    downloaded into pageable memory, and stay equal after unregistering."""
    rng = np.random.Generator(np.random.PCG64(41))
    t = _setup(ctx, rng, 31, 60, 9, 9, 4, 3, 3000)
    L = ctx.lib
    s = ctypes.c_uint64()
    ctx.check(L.slgpu_matrix_pattern_serial(ctx.h, t["h"], ctypes.byref(s)))
    assert s.value == 0
    A0, D0 = _process(ctx, t, abi.PREC_FP64)
    ctx.check(L.slgpu_matrix_pattern_serial(ctx.h, t["h"], ctypes.byref(s)))
    s0 = s.value
    assert s0 > 0
    _process(ctx, t, abi.PREC_FP64)
    ctx.check(L.slgpu_matrix_pattern_serial(ctx.h, t["h"], ctypes.byref(s)))
    assert s.value == s0

    buf = np.zeros(A0.size + 1024)
    ctx.check(L.slgpu_host_register(ctx.h, buf.ctypes.data, buf.nbytes))
    D = np.zeros(max(1, D0.size))
    ctx.check(L.slgpu_matrix_download_values(ctx.h, t["h"], abi.f64p(buf), abi.f64p(D)))
    assert np.array_equal(buf[: A0.size], A0) and np.array_equal(D[: D0.size], D0)
    ctx.check(L.slgpu_host_unregister(ctx.h, buf.ctypes.data))
    buf[:] = 0
    ctx.check(L.slgpu_matrix_download_values(ctx.h, t["h"], abi.f64p(buf), abi.f64p(D)))
    assert np.array_equal(buf[: A0.size], A0)

    t["con"] = t["con"].copy()
    t["con"][::5] ^= 1
    _process(ctx, t, abi.PREC_FP64)
    ctx.check(L.slgpu_matrix_pattern_serial(ctx.h, t["h"], ctypes.byref(s)))
    assert s.value != s0


def test_shared_address_arrays(ctx):
    """A group added twice with the same host address arrays (the second copy
    with other term scales), with slgpu_matrix_share_addresses on and off:
    the same CSR values bit for bit and the same pattern serial (addresses are
    hashed by content either way)."""
    rng = np.random.Generator(np.random.PCG64(43))
    L = ctx.lib
    gb, xyz, conn = S.group(rng, nelem_grid=40, ntf=9, ndof=9, nterms=4, ngp1=3, norient=2, ndests=2, ndofs=3000)
    g1 = gb.g
    g1.mesh = 33
    ctx.check(L.slgpu_mesh_set_nodes(ctx.h, 33, xyz.size // 3, abi.f64p(xyz)))
    ctx.check(L.slgpu_mesh_set_elements(ctx.h, 33, 3, 4, conn.size // 4, abi.i32p(conn)))
    g2 = abi.Group.from_buffer_copy(g1)
    terms2 = (abi.Term * g1.nterms)(*[abi.Term(g1.terms[t].tf_table, g1.terms[t].dof_table, g1.terms[t].coef_node, 0,
                                               0.5 + t) for t in range(g1.nterms)])
    g2.terms = terms2
    con = (rng.random(3000) < 0.1).astype(np.uint8)
    out = {}
    for share in (0, 1):
        h = ctypes.c_int()
        ctx.check(L.slgpu_matrix_create(ctx.h, 3000, ctypes.byref(h)))
        ctx.check(L.slgpu_matrix_share_addresses(ctx.h, h, share))
        ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g1), None))
        ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g2), None))
        A, D = _process(ctx, dict(h=h.value, con=con), abi.PREC_FP64)
        s = ctypes.c_uint64()
        ctx.check(L.slgpu_matrix_pattern_serial(ctx.h, h, ctypes.byref(s)))
        out[share] = (A, D, s.value)
        ctx.check(L.slgpu_matrix_destroy(ctx.h, h))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


@pytest.mark.parametrize("per_row,ndof,ndofs", [(1, 1, 50), (21, 1, 400), (22, 2, 400), (43, 3, 300), (5461, 1, 9000), (5462, 1, 9000),
                                                (700, 7, 60), (150, 33, 6000)])
def test_pattern_row_sizes(ctx, per_row, ndof, ndofs):
    """Rows with few to many COO entries, up to and beyond the most that the
    row-by-row pattern takes, with repeated columns, dropped and constrained
    ones, and two destinations: CSR structure equal to the oracle's, values
    within 1e-12 of the sums of magnitudes."""
    import os
    import sys

    sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
    import slref

    rng = np.random.Generator(np.random.PCG64(per_row + 7 * ndof))
    grid = int(np.ceil(np.sqrt(per_row))) + 1
    gb, xyz, conn = S.group(rng, nelem_grid=grid, ntf=2, ndof=ndof, nterms=2, ngp1=2, norient=1, ndests=2, ndofs=ndofs)
    g = gb.g
    # Test function 0 of the first per_row elements meets row 3; the others spread.
    tf = np.ctypeslib.as_array(g.dests[0].tfaddr, (2, g.nelem))
    tf[0, :] = -1
    tf[0, :per_row] = 3
    con = (rng.random(ndofs) < 0.1).astype(np.uint8)
    con[3] = 0
    ref = slref.matrix([g], xyz, [conn], ndofs, con)
    mag = slref.matrix([g], xyz, [conn], ndofs, con, absmode=True)
    L = ctx.lib
    ctx.check(L.slgpu_mesh_set_nodes(ctx.h, 41, xyz.size // 3, abi.f64p(xyz)))
    ctx.check(L.slgpu_mesh_set_elements(ctx.h, 41, 3, 4, conn.size // 4, abi.i32p(conn)))
    g.mesh = 41
    h = ctypes.c_int()
    ctx.check(L.slgpu_matrix_create(ctx.h, ndofs, ctypes.byref(h)))
    ctx.check(L.slgpu_matrix_add_group(ctx.h, h, ctypes.byref(g), None))
    info = abi.CsrInfo()
    ctx.check(L.slgpu_matrix_process(ctx.h, h, con.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), abi.PREC_FP64, ctypes.byref(info)))
    out = {k: np.zeros(max(1, n), t) for k, n, t in (("Arows", info.nA + 1, np.int32), ("Acols", info.nnzA, np.int32),
                                                     ("Avals", info.nnzA, np.float64), ("Drows", info.nA + 1, np.int32),
                                                     ("Dcols", info.nnzD, np.int32), ("Dvals", info.nnzD, np.float64))}
    ctx.check(L.slgpu_matrix_download(ctx.h, h, *[abi.i32p(v) if v.dtype == np.int32 else abi.f64p(v) for v in out.values()]))
    ctx.check(L.slgpu_matrix_destroy(ctx.h, h))
    for k in ("Arows", "Acols", "Drows", "Dcols"):
        assert np.array_equal(out[k][: ref[k].size], ref[k]), f"{k} differs"
    for k in ("Avals", "Dvals"):
        err = np.abs(out[k][: ref[k].size] - ref[k]) / np.maximum(mag[k], 1e-300)
        assert not err.size or err.max() <= 1e-12, f"{k}: {err.max():.3e}"


def test_graph_follows_unit_multipliers(tmp_path):
    """Destination multipliers that are all 1 when the step is captured and
    then are not: the warp value kernel, which takes multipliers of 1 from the
    launch, is captured anew.  Doubled multipliers give exactly doubled values,
    and the first values come back with the first multipliers."""
    import os
    import subprocess
    import sys

    code = """
import sys
import numpy as np
from sparselizard_b200 import abi
import test_gpu_graphs as T
ctx = abi.Context(0)
t = T._setup(ctx, np.random.Generator(np.random.PCG64(51)), 61, 30, 9, 9, 2, 2, 900)
n, out = t["ndests"], {}
for k, mult in enumerate([1.0] * 4 + [2.0] * 4 + [1.0] * 2):
    ctx.check(ctx.lib.slgpu_matrix_set_scales(ctx.h, t["h"], 0, None, abi.f64p(np.full(n, mult))))
    out["A%d" % k], out["D%d" % k] = T._process(ctx, t, abi.PREC_FP64)
assert ctx.lib.slgpu_graph_launches(ctx.h) >= 4
np.savez(sys.argv[1], **out)
"""
    here = os.path.dirname(os.path.abspath(__file__))
    out = str(tmp_path / "m.npz")
    env = dict(os.environ, SLGPU_ROW_KERNEL="warp", PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
    subprocess.run([sys.executable, "-c", code, out], env=env, check=True, timeout=300)
    r = np.load(out)
    for b in "AD":
        assert np.abs(r[b + "0"]).max() > 0
        for k in range(10):
            assert np.array_equal(r[f"{b}{k}"], r[b + "0"] * (2.0 if 4 <= k < 8 else 1.0)), f"{b}, call {k}"


def test_float_value_kernels_agree(tmp_path):
    """FP32-level steps through the warp kernels with windows of incidences
    across rows and per row, each forced in its own process: the same values
    bit for bit.  Rows of one to thousands of incidences, 1 to 31 rows a warp,
    widths up to and above a warp, repeated addresses, multipliers that are and
    are not 1."""
    import os
    import subprocess
    import sys

    code = """
import sys
import numpy as np
from sparselizard_b200 import abi
import test_gpu_graphs as T
ctx, out = abi.Context(0), {}
for k, (grid, ntf, ndof, ndofs) in enumerate([(9, 8, 8, 40), (60, 9, 9, 3000), (150, 8, 8, 100000), (260, 8, 8, 400000), (30, 8, 40, 4000),
                                              (40, 8, 32, 9000), (40, 8, 33, 9000)]):
    t = T._setup(ctx, np.random.Generator(np.random.PCG64(63 + k)), k, grid, ntf, ndof, 1, 2, ndofs)
    for mult in ([1.0, 1.0], [3.0, -2.5]):
        ctx.check(ctx.lib.slgpu_matrix_set_scales(ctx.h, t["h"], 0, None, abi.f64p(np.array(mult))))
        out["%d_%g_A" % (k, mult[0])], out["%d_%g_D" % (k, mult[0])] = T._process(ctx, t, abi.PREC_FP32)
np.savez(sys.argv[1], **out)
"""
    here = os.path.dirname(os.path.abspath(__file__))
    res = {}
    for k in ("warp", "row"):
        out = str(tmp_path / f"{k}.npz")
        env = dict(os.environ, SLGPU_ROW_KERNEL=k, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here)]))
        subprocess.run([sys.executable, "-c", code, out], env=env, check=True, timeout=300)
        res[k] = np.load(out)
    for key in res["warp"].files:
        a, b = res["warp"][key], res["row"][key]
        assert np.all(np.isfinite(a)) and np.abs(a).max() > 0 and np.array_equal(a, b), key
