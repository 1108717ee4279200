"""The line forms of the BP5/BP6 operators on Hex3D where a block serves several
(element, field) slots: permuted partial element lists (one value per node) and
four packed right-hand sides, against the FP64 oracle; and stored factors of any
alignment.

1e-12 relative in FP64 as elsewhere (sums of at most 16 terms per 1D step);
2e-5 in FP32, the bar of the other FP32 operators."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7, 9, 12, 15])
@pytest.mark.parametrize("affine,nf", [(False, 1), (True, 1), (False, 3), (True, 3)])
def test_hex_permuted_subset(gpu, oracle, monkeypatch, N, affine, nf):
    monkeypatch.setenv("BP_AX_VARIANT", "line")
    om = oracle.Mesh(3, 2, 2, N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    gm = gpu.Mesh(3, 2, 2, N=N, affine=affine, Nfields=nf, pert=0.0 if affine else 0.1)
    q = 2 * oracle.random(5, om.Ngather) - 1
    want = om.ax(q).reshape(gm.E, -1)
    els = np.array([10, 3, 7, 0, 11], np.int32)
    dq, dA = gpu.DeviceBuffer.from_host(q), gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan))
    de = gpu.DeviceBuffer.from_host(els)
    gpu.ax_hex3d(gm, dq, dA, elementList=de.ptr, Nelements=els.size)
    got = dA.download().reshape(gm.E, -1)
    assert np.all(np.isnan(got[np.setdiff1d(np.arange(gm.E), els)]))
    assert _rel(got[els], want[els]) < 1e-12


# Stored factors aligned to one element only are read one by one by the pencil
# form, whatever form is forced or recorded for aligned calls, and record nothing.
@pytest.mark.parametrize("variant", ["", "line"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,nf", [(4, 1), (7, 1), (7, 3)])
def test_factors_aligned_to_one_element(gpu, oracle, monkeypatch, N, nf, dtype, variant):
    if variant:
        monkeypatch.setenv("BP_AX_VARIANT", variant)
    om, gm = oracle.Mesh(3, 2, 2, N, Nfields=nf, pert=0.1), gpu.Mesh(3, 2, 2, N=N, Nfields=nf, pert=0.1)
    d, v = gpu.AxDesc(5 if nf == 1 else 6, N, 0, nf), gm.view
    q = (2 * oracle.random(5, om.Ngather) - 1).astype(dtype)
    ops = {k: gpu.DeviceBuffer.from_host(gm.array(k).astype(dtype)) for k in ("wJ", "gllw", "D")}
    g = gm.array("ggeo").astype(dtype)
    bufs = [gpu.DeviceBuffer.from_host(np.concatenate([np.zeros(off, dtype), g])) for off in (0, 1)]
    dq, f = gpu.DeviceBuffer.from_host(q), gpu.lib().bp_ax_hex3d if dtype == np.float64 else gpu.lib().bp_ax_hex3d_f32
    out, forms = [], []
    for off, b in enumerate(bufs):
        dA = gpu.DeviceBuffer.from_host(np.full(gm.NL, np.nan, dtype))
        gpu._check(f(gpu.ctypes.byref(d), gm.E, v.elementList, v.GlobalToLocal, ops["wJ"].ptr,
                     b.ptr + off * g.itemsize, ops["gllw"].ptr, ops["D"].ptr, 1.0, dq.ptr, dA.ptr, None))
        out.append(dA.download().astype(np.float64))
        forms.append(gpu.tune_report(0, N, nf, 0, g.itemsize, 1, 0, gm.E)[0])
    want = om.ax(q.astype(np.float64))
    for o in out:
        assert _rel(o, want) < (1e-12 if dtype == np.float64 else 2e-5)
    assert forms[0] == forms[1]


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7, 8, 10])
def test_packed_lines(gpu, oracle, monkeypatch, N):
    monkeypatch.setenv("BP_AX_VARIANT", "line")
    om, gm = oracle.Mesh(3, 3, 2, N, pert=0.1), gpu.Mesh(3, 3, 2, N=N, pert=0.1)
    v, ng = gm.view, gm.E * gm.Np
    ops = {}
    for name, n in (("wJ", ng), ("ggeo", 6 * ng), ("gllw", gm.Nq), ("D", gm.Nq ** 2)):
        ops[name] = gpu.DeviceBuffer(n, np.float32)
        gpu.convert_f64_f32(getattr(v, name), n, ops[name])
    q = np.stack([2 * oracle.random(k, om.Ngather) - 1 for k in range(4)], 1).astype(np.float32)
    dq = gpu.DeviceBuffer.from_host(q)
    dA = gpu.DeviceBuffer.from_host(np.full(4 * gm.NL, np.nan, np.float32))
    gpu.ax_hex3d_f32_multi(gm, 4, dq, dA, ops)
    got = dA.download().reshape(-1, 4).astype(np.float64)
    for k in range(4):
        assert _rel(got[:, k], om.ax(q[:, k].astype(np.float64))) < 2e-5
