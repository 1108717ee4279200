"""The over-integrated operators (ax_cub_kernel) where a block serves several
(element, field) slots: element counts that leave the last block partly empty,
permuted element lists, three fields, and q.Aq inside CG with one partial per
block (more blocks than elements with three fields).

Against the FP64 oracle; 1e-12 relative as for the other operators (the sums
are up to 17 terms per 1D step, six steps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


# G points per direction 2..17; slots per block 24, 21, 6, 5, 2, 1 (stiffness), 24, 21, 12, 5, 3, 2, 1 (mass)
@pytest.mark.parametrize("N,affine", [(1, True), (1, False), (2, False), (3, False), (4, False), (5, False), (6, False),
                                      (7, False), (7, True), (9, True), (12, False), (14, False)])
@pytest.mark.parametrize("bpn", [1, 2, 3, 4])
def test_permuted_subset_and_partial_blocks(gpu, oracle, N, affine, bpn):
    nf = 1 if bpn % 2 else 3
    om = oracle.Mesh(3, 2, 3, N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    gm = gpu.Mesh(3, 2, 3, N=N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    q = 2 * oracle.random(5, om.Ngather) - 1
    want = om.ax(q, 1.0, bpn).reshape(gm.E, -1)
    els = np.array([16, 3, 11, 0, 7, 17, 5], np.int32)
    dq, dA = gpu.DeviceBuffer.from_host(q), gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan))
    de = gpu.DeviceBuffer.from_host(els)
    v, c = gm.view, gm.cubature()
    d = gpu.AxDesc(bpn, N, int(affine), nf)
    gpu._check(gpu.lib().bp_ax_cub_hex3d(gpu.ctypes.byref(d), els.size, de.ptr, v.GlobalToLocal, c.cubwJ, c.cubggeo,
                                         c.cubD, c.cubInterp, c.invV, c.MM, 1.0, dq.ptr, dA.ptr, None))
    got = dA.download().reshape(gm.E, -1)
    rest = np.setdiff1d(np.arange(gm.E), els)
    assert np.all(np.isnan(got[rest]))          # only the listed elements are written
    assert _rel(got[els], want[els]) < 1e-12


@pytest.mark.parametrize("bpn,N", [(2, 1), (4, 1), (4, 6), (2, 7)])
def test_three_field_cg_has_room_for_its_partials(gpu, oracle, bpn, N):
    om = oracle.Mesh(4, 4, 3, N, Nfields=3, pert=0.1)
    gm = gpu.Mesh(4, 4, 3, N=N, Nfields=3, pert=0.1)
    b = om.rhs_random(3)[1]
    S = gpu.BP(gm, bp=bpn, precon="JACOBI")
    x = gpu.DeviceBuffer.from_host(np.zeros(om.Ngather))
    st, hr, _ = S.solve(x, gpu.DeviceBuffer.from_host(b), tol=0.0, maxit=4)
    _, _, _, ho, _ = om.cg(b, 1.0, 0.0, 4, precon=True, bp=bpn)
    assert st.iterations == 4
    assert np.max(np.abs(hr - ho) / ho) < 1e-10
