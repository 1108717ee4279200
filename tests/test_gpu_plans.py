"""Operators whose form or tile plan a rule picks by the number of elements, in
every form and plan, with the plan asserted: Quad2D on both sides of its rule
(line and node form, all degrees, FP64 and FP32) and inside CG; the simplex
operator's tiles per warp, warps along the nodes and row split.

Against numpy on the mesh's own factors and matrices: an oracle's factors differ
from the library's by the cancellation in the coordinate derivatives, which is
no property of the operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _plan(gpu, dim, simplex, N, affine, nf, n, precision_bytes=8):
    p = np.zeros(4, np.int32)
    gpu._check(gpu.lib().bp_test_operator_plan(dim, int(simplex), N, int(affine), nf, precision_bytes, n, p.ctypes.data))
    return tuple(int(v) for v in p)


def _gathered(gm, q):
    ids = gm.array("GlobalToLocal")
    return np.where(ids >= 0, q[np.maximum(ids, 0)], 0.0)


def _quad_reference(gm, q):
    nf, E, n = gm.Nfields, gm.E, gm.Nq
    D, w = gm.array("D").reshape(n, n), gm.array("gllw")
    g, J = gm.array("ggeo").reshape(E, -1, 3), gm.array("wJ").reshape(E, -1)
    if gm.affine:
        ww = np.outer(w, w).reshape(-1)
        g, J = g * ww[None, :, None], J * ww[None, :]
    g, J = g.reshape(E, 1, n, n, 3), J.reshape(E, 1, n, n)
    u = _gathered(gm, q).reshape(E, nf, n, n)
    ur, us = u @ D.T, D @ u
    fr, fs = g[..., 0] * ur + g[..., 1] * us, g[..., 1] * ur + g[..., 2] * us
    return (J * u + fr @ D + D.T @ fs).reshape(E, -1)


def _quad_mesh(gpu, N, affine, nf, line):
    """The smallest box of nx x (nx + 1) elements that takes the line form in both precisions, or 3 x 2."""
    nx, ny = 3, 2
    if line:
        while not all(_plan(gpu, 2, False, N, affine, nf, nx * ny, b)[0] for b in (8, 4)):
            nx += 1
            ny = nx + 1
    gm = gpu.Mesh(nx, ny, 1, N=N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1, dim=2)
    assert all(_plan(gpu, 2, False, N, affine, nf, gm.E, b)[0] == int(line) for b in (8, 4))
    return gm


# FP64: two sums of Nq terms in each direction, 4 Nq 2^-53 < 1e-14 on terms that
# cancel to a tenth at the most; FP32 2e-5, the bar of the other FP32 operators
@pytest.mark.parametrize("line", [False, True])
@pytest.mark.parametrize("N", range(1, 16))
@pytest.mark.parametrize("affine,nf", [(False, 1), (True, 1), (False, 2), (True, 2)])
def test_quad_forms(gpu, oracle, N, affine, nf, line):
    gm = _quad_mesh(gpu, N, affine, nf, line)
    q = (2 * oracle.random(5, gm.Ngather) - 1).astype(np.float32).astype(np.float64)
    want = _quad_reference(gm, q)
    dq, dA = gpu.DeviceBuffer.from_host(q), gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan))
    gpu.ax_hex3d(gm, dq, dA)
    assert _rel(dA.download().reshape(gm.E, -1), want) < 1e-13
    ops = {k: gpu.DeviceBuffer.from_host(gm.array(k).astype(np.float32)) for k in ("wJ", "ggeo", "gllw", "D")}
    dA = gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan, np.float32))
    gpu.ax_hex3d_f32(gm, gpu.DeviceBuffer.from_host(q.astype(np.float32)), dA, ops)
    assert _rel(dA.download().reshape(gm.E, -1).astype(np.float64), want) < 2e-5


# a permuted list without the last elements, so that the last block is partly empty
@pytest.mark.parametrize("N,nf", [(1, 2), (2, 1), (4, 1), (7, 1), (7, 2), (10, 1), (15, 2)])
def test_quad_line_form_on_a_permuted_subset(gpu, oracle, N, nf):
    gm = _quad_mesh(gpu, N, True, nf, True)
    gm = gpu.Mesh(gm.nx + 2, gm.ny + 2, 1, N=N, affine=True, Nfields=nf, dim=2)
    els = np.random.default_rng(N).permutation(gm.E)[:gm.E - 5].astype(np.int32)
    assert _plan(gpu, 2, False, N, True, nf, els.size)[0] == 1
    q = 2 * oracle.random(5, gm.Ngather) - 1
    dA = gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan))
    gpu.ax_hex3d(gm, gpu.DeviceBuffer.from_host(q), dA, elementList=gpu.DeviceBuffer.from_host(els).ptr,
                 Nelements=els.size)
    got, want = dA.download().reshape(gm.E, -1), _quad_reference(gm, q)
    assert np.all(np.isnan(got[np.setdiff1d(np.arange(gm.E), els)]))
    assert _rel(got[els], want[els]) < 1e-13


# p.Ap of the line form: 1e-10 per iteration as elsewhere, and the mixed solve's own bar
@pytest.mark.parametrize("N,affine,nf", [(2, False, 1), (5, True, 2), (7, False, 1)])
def test_quad_line_form_inside_cg(gpu, oracle, N, affine, nf):
    gm = _quad_mesh(gpu, N, affine, nf, True)
    om = oracle.Mesh(gm.nx, gm.ny, 0, N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1, dim=2)
    b = om.rhs_random(0)[1]
    x = gpu.DeviceBuffer.from_host(np.zeros(om.Ngather))
    st, hr, _ = gpu.BP(gm, precon="JACOBI").solve(x, gpu.DeviceBuffer.from_host(b), tol=0.0, maxit=10)
    ho = om.cg(b, 1.0, 0.0, 10, precon=True)[3]
    assert st.iterations == 10 and np.max(np.abs(hr - ho) / ho) < 1e-10
    x = gpu.DeviceBuffer.from_host(np.zeros(om.Ngather))
    gpu.BP(gm, precon="JACOBI", precision="MIXED").solve(x, gpu.DeviceBuffer.from_host(b), tol=1e-8, maxit=20000)
    assert np.linalg.norm(b - om.operator(x.download())) <= 1.0001e-8 * np.linalg.norm(b)


def _simplex_reference(gm, q):
    """sum_c f_c(e) X_c q_e over the stiffness matrices and MM (stored node-fastest:
    row k of an array holds X(:, k))."""
    C = 3 if gm.dim == 2 else 6
    S = gm.array("S").reshape(C, gm.Np, gm.Np)
    g, u = gm.array("ggeo").reshape(gm.E, C), _gathered(gm, q).reshape(gm.E, gm.Np)
    out = gm.array("wJ").reshape(gm.E, 1) * (u @ gm.array("MM").reshape(gm.Np, gm.Np))
    for c in range(C):
        out += g[:, c:c + 1] * (u @ S[c])
    return out


# (dim, degree, cells per direction) and the 8-node tiles, 8-element tiles and warps
# along the nodes of the plan on 148 SMs.  The permuted list leaves elements out,
# and the last tile partly empty in the one list or the other.
PLANS = [(2, 3, 1, 1, 1, 1), (2, 6, 1, 1, 1, 2), (2, 9, 1, 1, 1, 4), (3, 2, 12, 1, 2, 2), (2, 6, 50, 1, 2, 4),
         (2, 3, 43, 2, 1, 1), (2, 6, 33, 2, 1, 2), (2, 13, 17, 2, 1, 4), (2, 3, 110, 2, 2, 1), (2, 6, 80, 2, 2, 2),
         (2, 9, 51, 2, 2, 4), (2, 5, 45, 3, 1, 1), (2, 7, 29, 3, 1, 2), (2, 10, 22, 3, 1, 4), (3, 3, 16, 3, 2, 1),
         (2, 8, 80, 3, 2, 2), (3, 8, 7, 3, 2, 4), (2, 13, 26, 4, 1, 4), (2, 6, 120, 4, 2, 1), (3, 8, 8, 4, 2, 2),
         (3, 9, 7, 4, 2, 4), (2, 7, 80, 5, 1, 1), (3, 9, 6, 5, 1, 2), (2, 15, 24, 5, 1, 4), (3, 4, 16, 5, 2, 1),
         (2, 10, 80, 5, 2, 2), (3, 10, 7, 5, 2, 4)]


def _simplex_mesh(gpu, dim, N, n):
    return gpu.Mesh(n, n, n if dim == 3 else 1, N=N, affine=True, dim=dim, simplex=True)


def _simplex_apply(gpu, gm, q, els):
    d, v = gpu.AxDesc(5, gm.N, 1, 1, gm.dim), gm.view
    f = gpu.lib().bp_ax_tri2d if gm.dim == 2 else gpu.lib().bp_ax_tet3d
    dq, dA = gpu.DeviceBuffer.from_host(q), gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan))
    de = gpu.DeviceBuffer.from_host(els)
    gpu._check(f(gpu.ctypes.byref(d), els.size, de.ptr, v.GlobalToLocal, v.wJ, v.ggeo, v.S, v.MM, 1.0, dq.ptr, dA.ptr,
                 None))
    return dA.download().reshape(gm.E, -1)


# A sum over k of Np terms and one over c of at most 7: (Np + 7) 2^-53 of the terms'
# absolute sum in either order of summation, and that sum beside the result in the
# maximum norm: both from the same matrices.
def _simplex_bound(gm, q):
    C = 3 if gm.dim == 2 else 6
    u = np.abs(_gathered(gm, q).reshape(gm.E, gm.Np))
    a = np.abs(gm.array("wJ")).reshape(gm.E, 1) * (u @ np.abs(gm.array("MM").reshape(gm.Np, gm.Np)))
    for c in range(C):
        a += np.abs(gm.array("ggeo").reshape(gm.E, C)[:, c:c + 1]) * (u @ np.abs(gm.array("S").reshape(C, gm.Np, gm.Np)[c]))
    return 2 * (gm.Np + 7) * 2.0 ** -53 * a


@pytest.mark.parametrize("dim,N,n,mt,nt,wm", PLANS)
def test_simplex_plans(gpu, dim, N, n, mt, nt, wm):
    gm = _simplex_mesh(gpu, dim, N, n)
    rng = np.random.default_rng(N)
    q = 2 * rng.random(gm.Ngather) - 1
    want, bound = _simplex_reference(gm, q), _simplex_bound(gm, q)
    full, part = np.arange(gm.E, dtype=np.int32), rng.permutation(gm.E)[:gm.E - gm.E // 50 - 1].astype(np.int32)
    plan = _plan(gpu, dim, True, N, True, 1, gm.E)
    sms = gpu.ctypes.c_int()
    gpu._check(gpu.lib().bp_device_info(None, 0, gpu.ctypes.byref(sms)))
    if sms.value == 148:
        assert plan[:3] == (mt, nt, wm)
    for els in (full, part):
        got = _simplex_apply(gpu, gm, q, els)
        assert np.all(np.isnan(got[np.setdiff1d(full, els)]))
        assert np.all(np.abs(got[els] - want[els]) <= bound[els])


def test_simplex_plans_cover_every_tile_shape_and_both_row_splits(gpu):
    shapes = {p[3:5] for p in PLANS}
    assert shapes == {(mt, nt) for mt in range(1, 6) for nt in (1, 2)}
    gy = [_plan(gpu, d, True, N, True, 1, 2 * n * n if d == 2 else 6 * n ** 3)[3] for d, N, n, *_ in PLANS]
    assert min(gy) == 1 and sum(g > 1 for g in gy) >= 5


# p.Ap with several m-tiles, two n-tiles and a row split: history against the oracle's
@pytest.mark.parametrize("dim,N,n", [(2, 3, 90), (2, 10, 22), (3, 4, 14), (3, 8, 7)])
def test_simplex_plans_inside_cg(gpu, dim, N, n):
    gm = _simplex_mesh(gpu, dim, N, n)
    S = gpu.BP(gm, precon="JACOBI")
    b, dinv = S.rhs("RANDOM", 0).download(), 1.0 / S.diagonal().download()
    x = gpu.DeviceBuffer.from_host(np.zeros(gm.Ngather))
    st, hr, _ = S.solve(x, gpu.DeviceBuffer.from_host(b), tol=0.0, maxit=6)
    rows, cols = gm.array("rowStarts"), gm.array("colIds")
    r, p, ho = b.copy(), None, []
    for k in range(6):
        z = dinv * r
        rz = r @ z
        p = z if p is None else z + rz / rz0 * p
        Ap = np.add.reduceat(_simplex_reference(gm, p).reshape(-1)[cols], rows[:-1])
        r, rz0 = r - rz / (p @ Ap) * Ap, rz
        ho.append(np.linalg.norm(r))
    assert st.iterations == 6 and np.max(np.abs(hr - ho) / ho) < 1e-10
