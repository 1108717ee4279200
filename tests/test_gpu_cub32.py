"""The over-integrated operators in FP32 (ax_cub_kernel, the inner operator of the
mixed-precision solves): all four forms over the degrees at which the slots per
block, the unrolling and the shared-memory strides change, partly empty last
blocks and permuted partial lists; and the mixed
CG, whose p.Ap comes from one partial per block.

Against the FP64 oracle at the bar of the other FP32 operators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _f32_ops(gpu, gm):
    c = gm.cubature()
    nc = gm.E * (1 if gm.affine else c.cubNp)
    nq2, g2 = gm.Nq * gm.Nq, c.cubNq * c.cubNq
    sizes = {"cubwJ": nc, "cubggeo": 6 * nc, "cubD": nq2 if gm.affine else g2,
             "cubInterp": 0 if gm.affine else c.cubNq * gm.Nq, "invV": nq2 if gm.affine else 0,
             "MM": nq2 if gm.affine else 0}
    ops = {}
    for name, n in sizes.items():
        ops[name] = gpu.DeviceBuffer(max(n, 1), np.float32)
        if n:
            gpu.convert_f64_f32(getattr(c, name), n, ops[name])
    return ops


def _apply(gpu, gm, bpn, ops, dq, dA, elist=None, nel=None):
    d = gpu.AxDesc(bpn, gm.N, int(gm.affine), gm.Nfields)
    v = gm.view
    gpu._check(gpu.lib().bp_ax_cub_hex3d_f32(gpu.ctypes.byref(d), gm.E if nel is None else nel,
                                             v.elementList if elist is None else elist.ptr, v.GlobalToLocal,
                                             ops["cubwJ"].ptr, ops["cubggeo"].ptr, ops["cubD"].ptr,
                                             ops["cubInterp"].ptr, ops["invV"].ptr, ops["MM"].ptr, 1.0, dq.ptr,
                                             dA.ptr, None))


# 10^3 at p=7: several blocks per SM; most of the others leave the last block partly empty
@pytest.mark.parametrize("nx,ny,nz,N", [(3, 2, 2, 7), (5, 5, 5, 7), (10, 10, 10, 7), (4, 3, 3, 5), (3, 3, 2, 3),
                                        (2, 2, 2, 11), (2, 1, 1, 13), (3, 3, 3, 1)])
def test_curved_stiffness_matches_oracle(gpu, oracle, nx, ny, nz, N):
    om = oracle.Mesh(nx, ny, nz, N, pert=0.1)
    gm = gpu.Mesh(nx, ny, nz, N=N, pert=0.1)
    q = (2 * oracle.random(8, om.Ngather) - 1).astype(np.float32)
    dA = gpu.DeviceBuffer.from_host(np.full(om.NL, np.nan, np.float32))
    _apply(gpu, gm, 3, _f32_ops(gpu, gm), gpu.DeviceBuffer.from_host(q), dA)
    assert _rel(dA.download().astype(np.float64), om.ax(q.astype(np.float64), 1.0, 3)) < 2e-5


# a partial element list in shuffled order: exactly the listed elements are written
@pytest.mark.parametrize("bpn", [1, 2, 3, 4])
@pytest.mark.parametrize("N,affine", [(1, True), (1, False), (2, False), (3, False), (4, True), (5, False), (5, True),
                                      (6, False), (7, False), (7, True), (9, False), (10, False), (11, True),
                                      (12, False), (13, True), (14, False), (15, True)])
def test_forms_on_a_permuted_subset(gpu, oracle, bpn, N, affine):
    nf = 1 if bpn % 2 else 3
    om = oracle.Mesh(3, 2, 3, N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    gm = gpu.Mesh(3, 2, 3, N=N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    q = (2 * oracle.random(9, om.Ngather) - 1).astype(np.float32)
    sub = np.random.default_rng(3).permutation(gm.E)[:7].astype(np.int32)
    dA = gpu.DeviceBuffer.from_host(np.full(om.NL, np.nan, np.float32))
    _apply(gpu, gm, bpn, _f32_ops(gpu, gm), gpu.DeviceBuffer.from_host(q), dA, gpu.DeviceBuffer.from_host(sub), sub.size)
    got, want = dA.download().reshape(gm.E, -1), om.ax(q.astype(np.float64), 1.0, bpn).reshape(gm.E, -1)
    assert np.all(np.isnan(got[np.setdiff1d(np.arange(gm.E), sub)]))
    assert _rel(got[sub].astype(np.float64), want[sub]) < 2e-5


@pytest.mark.parametrize("bpn,N,affine,n", [(3, 7, False, (6, 6, 5)), (1, 4, False, (6, 5, 4)), (3, 5, True, (6, 5, 4)),
                                            (4, 6, False, (4, 3, 3))])
def test_mixed_solve_reaches_tolerance(gpu, oracle, bpn, N, affine, n):
    nf, pert = (1 if bpn % 2 else 3), 0.0 if affine else 0.1
    om, gm = oracle.Mesh(*n, N, affine=affine, Nfields=nf, pert=pert), gpu.Mesh(*n, N=N, affine=affine, Nfields=nf, pert=pert)
    b = om.rhs_random(0)[1]
    x = gpu.DeviceBuffer.from_host(np.zeros(gm.Ngather))
    st, _, _ = gpu.BP(gm, bp=bpn, precon="JACOBI", precision="MIXED").solve(x, gpu.DeviceBuffer.from_host(b), tol=1e-8,
                                                                           maxit=5000)
    assert np.linalg.norm(b - om.operator(x.download(), bp=bpn)) <= 1.0001e-8 * np.linalg.norm(b)
    x64 = gpu.DeviceBuffer.from_host(np.zeros(gm.Ngather))
    s64, _, _ = gpu.BP(gm, bp=bpn, precon="JACOBI").solve(x64, gpu.DeviceBuffer.from_host(b), tol=1e-8, maxit=5000)
    assert abs(st.iterations - s64.iterations) <= 0.02 * s64.iterations + 3   # the FP64 recursion's count
    assert _rel(x.download(), x64.download()) < 1e-6
