"""Operators whose form or tile plan a rule picks by the number of elements, in
every form and plan, with the plan asserted: Quad2D on both sides of its rule
(line and node form, all degrees, FP64 and FP32) and inside CG.

Against numpy on the mesh's own factors and matrices: an oracle's factors differ
from the library's by the cancellation in the coordinate derivatives, which is
no property of the operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _plan(gpu, dim, simplex, N, affine, nf, n):
    p = np.zeros(4, np.int32)
    gpu._check(gpu.lib().bp_test_operator_plan(dim, int(simplex), N, int(affine), nf, n, p.ctypes.data))
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
    """The smallest box of nx x (nx + 1) elements that takes the line form, or 3 x 2."""
    nx, ny = 3, 2
    if line:
        while not _plan(gpu, 2, False, N, affine, nf, nx * ny)[0]:
            nx += 1
            ny = nx + 1
    gm = gpu.Mesh(nx, ny, 1, N=N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1, dim=2)
    assert _plan(gpu, 2, False, N, affine, nf, gm.E)[0] == int(line)
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
