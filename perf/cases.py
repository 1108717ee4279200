"""The work that a user of the library has it do, as cases that can be timed.

Element operators as the BK benchmarks call them, the assembled operator, CG
solves in FP64 and in mixed precision, and the batched solver, each through the
public Python entry points, over the degrees 1..15, the element types, affine
and stored factors and the field counts that the BP1..BP6 problems take.
Meshes are the library's boxes, their interior vertices perturbed by 0.1 h with
a seed of the case's own (curved elements) or undeformed (affine)."""
import math

import numpy as np
import torch

import benchparanumal_b200 as bp

LAMBDA = 1.0
TOL = 1e-8


def listed():
    return [
        # one assembled operator application on a small mesh: a smoother's or an outer solver's call, where launches count
        {"name": "operator-small", "kind": "operator", "bp": 5, "el": "hex", "N": 4, "nx": 6, "ny": 5, "nz": 7, "affine": False},
        # the headline operator of the benchmark: BK5 at degree 7 on 40^3 curved elements
        {"name": "bk5-p7-large", "kind": "ax", "bp": 5, "el": "hex", "N": 7, "nx": 40, "ny": 40, "nz": 40, "affine": False},
        # an odd number of nodes per direction on a ragged box
        {"name": "bk5-p10-ragged", "kind": "ax", "bp": 5, "el": "hex", "N": 10, "nx": 19, "ny": 23, "nz": 17, "affine": False},
        # the highest degree, three fields, affine elements (the BP6 configuration of the benchmark, smaller)
        {"name": "bk6-p15-affine", "kind": "ax", "bp": 6, "el": "hex", "N": 15, "nx": 14, "ny": 14, "nz": 14, "affine": True},
        # over-integrated mass matrix on curved elements
        {"name": "bk1-p7", "kind": "ax", "bp": 1, "el": "hex", "N": 7, "nx": 32, "ny": 32, "nz": 32, "affine": False},
        # over-integrated stiffness on curved elements (the BP3 configuration of the benchmark)
        {"name": "bk3-p7-large", "kind": "ax", "bp": 3, "el": "hex", "N": 7, "nx": 40, "ny": 40, "nz": 40, "affine": False},
        # over-integrated stiffness with three fields at a middle degree on a ragged box
        {"name": "bk4-p5-ragged", "kind": "ax", "bp": 4, "el": "hex", "N": 5, "nx": 21, "ny": 18, "nz": 23, "affine": False},
        # two dimensions: curved quadrilaterals
        {"name": "quad-p7", "kind": "ax", "bp": 5, "el": "quad", "N": 7, "nx": 700, "ny": 500, "nz": 1, "affine": False},
        # tetrahedra
        {"name": "tet-p4", "kind": "ax", "bp": 5, "el": "tet", "N": 4, "nx": 26, "ny": 25, "nz": 24, "affine": True},
        # the reference's own run on the small configuration: 100 CG iterations in FP64, Jacobi-preconditioned
        {"name": "cg-fp64-p4-small", "kind": "cg", "bp": 5, "el": "hex", "N": 4, "nx": 16, "ny": 16, "nz": 16, "affine": False},
        # one over-integrated problem solved from host arrays to 1e-8 in mixed precision
        {"name": "solve-bp3-mixed", "kind": "solve", "bp": 3, "el": "hex", "N": 6, "nx": 13, "ny": 14, "nz": 12, "affine": False},
        # four right-hand sides of one problem solved together to 1e-8 in mixed precision (the benchmark's step, smaller)
        {"name": "batch-bp5-4rhs", "kind": "batch", "bp": 5, "el": "hex", "N": 7, "nx": 22, "ny": 24, "nz": 23, "affine": False},
    ]


def draw(rng):
    kind = rng.choice(["ax"] * 9 + ["operator"] * 3 + ["cg"] * 2 + ["solve", "batch"])
    el = "hex" if kind in ("cg", "solve", "batch") else rng.choice(["hex"] * 6 + ["quad", "quad", "tri", "tet"])
    affine = rng.random() < 0.35
    if kind in ("cg", "batch"):
        b = 5
    elif kind == "solve":
        b = rng.choice([3, 5])
    elif el == "hex":
        b = rng.choice([1, 2, 3, 4, 5, 6])
    elif el == "quad":
        b = rng.choice([5, 6])
    else:
        b, affine = 5, True
    iterative = kind in ("cg", "solve", "batch")
    N = rng.randint(2, 9) if iterative else rng.randint(1, 10) if el == "tet" else rng.randint(1, 15)
    # unknowns per field, over the logarithm; elements per direction, unequal
    hi = {"cg": 4e6, "solve": 8e5, "batch": 6e5}.get(kind, {"hex": 1.2e7, "quad": 8e6}.get(el, 8e5)) / fields(b, el)
    lo = 2e5 if kind == "cg" else 3e3      # 100 iterations leave a mesh of this size unconverged
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    dim = 3 if el in ("hex", "tet") else 2
    n = (want ** (1.0 / dim)) / N
    side = [max(2, int(round(n * rng.uniform(0.85, 1.15)))) for _ in range(3)]
    return {"kind": kind, "bp": b, "el": el, "N": N, "nx": side[0], "ny": side[1], "nz": side[2] if dim == 3 else 1, "affine": affine}


# ---------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------
def fields(b, el):
    return (3 if el == "hex" else 2) if b % 2 == 0 else 1


def sizes(c):
    """Elements, nodes per element, fields, unknowns, quadrature points per direction."""
    N, nx, ny, nz = c["N"], c["nx"], c["ny"], c["nz"]
    nf = fields(c["bp"], c["el"])
    dim = 3 if c["el"] in ("hex", "tet") else 2
    E = nx * ny * (nz if dim == 3 else 1) * {"tri": 2, "tet": 6}.get(c["el"], 1)
    if c["el"] == "tri":
        Np = (N + 1) * (N + 2) // 2
    elif c["el"] == "tet":
        Np = (N + 1) * (N + 2) * (N + 3) // 6
    else:
        Np = (N + 1) ** dim
    Nd = (nx * N - 1) * (ny * N - 1) * ((nz * N - 1) if dim == 3 else 1) * nf
    return E, Np, nf, Nd


def ax_work(c, s):
    """(bytes of the stored operator data, flops) of one element operator with s-byte values."""
    E, Np, nf, _ = sizes(c)
    N, Nq, b = c["N"], c["N"] + 1, c["bp"]
    if c["el"] in ("tri", "tet"):
        m = 3 if c["el"] == "tri" else 6
        return E * (m + 1) * s, 2.0 * (m + 1) * Np * Np * E
    if c["el"] == "quad":
        pts = 1 if c["affine"] else Np
        return E * pts * 4 * s, E * nf * (8.0 * Nq ** 3 + 10 * Np)
    if b >= 5:
        pts = 1 if c["affine"] else Np
        return E * pts * 7 * s, E * nf * (12.0 * Nq ** 4 + 18 * Np)
    G = Nq if c["affine"] else Nq + 1
    pts = 1 if c["affine"] else G ** 3
    interp = 2.0 * (Nq ** 3 * G + Nq ** 2 * G ** 2 + Nq * G ** 3)
    if b <= 2:
        fl = (6.0 * Nq ** 4 + Np) if c["affine"] else 2 * interp + G ** 3
        return E * pts * s, E * nf * fl
    return E * pts * 7 * s, E * nf * (2 * interp + 12.0 * G ** 4 + 18 * G ** 3)


def iterations(c):
    """CG iterations to 1e-8: they grow as degree times elements per side."""
    return 4.8 * c["N"] * max(c["nx"], c["ny"], c["nz"])


def work(c):
    E, Np, nf, Nd = sizes(c)
    NL = E * Np * nf
    if c["kind"] == "ax":     # q and the factors in, the map, the element-local result out
        by, fl = ax_work(c, 8)
        return {"bytes": by + 8.0 * Nd + 4.0 * NL + 8.0 * NL, "flops": fl}
    if c["kind"] == "operator":   # the result assembled
        by, fl = ax_work(c, 8)
        return {"bytes": by + 16.0 * Nd + 4.0 * NL, "flops": fl + NL}
    # per iteration: the factors and the map, x, r and p in and out, the inverse diagonal in
    if c["kind"] == "cg":
        by, fl = ax_work(c, 8)
        return {"bytes": 100.0 * (by + 4.0 * NL + 7 * 8.0 * Nd), "flops": 100.0 * (fl + NL + 12.0 * Nd)}
    by, fl = ax_work(c, 4)
    rhs = 4 if c["kind"] == "batch" else 1
    it = iterations(c)
    return {"bytes": it * (by + 4.0 * NL + 4.0 * Nd + rhs * 6 * 4.0 * Nd), "flops": it * rhs * (fl + NL + 12.0 * Nd)}


def tolerance(c):
    # four times the largest distance from the FP64 torch results seen over listed and drawn cases
    if c["kind"] in ("ax", "operator"):
        return {"rel": 2e-15}
    if c["kind"] == "cg":      # 100 iterations that have not converged; the sums' order travels through them
        return {"rel": 1e-12}
    return {"rel": 1.5e-6}     # solved to a residual of 1e-8, times what the condition number makes of it


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
class _Array:
    def __init__(self, owner, ptr, n):
        self.owner = owner     # the memory lives as long as a tensor on it
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "<f8", "data": (int(ptr), False), "version": 2}


def view(buffer, n=None, ptr=None):
    """A torch tensor on the doubles of a device buffer, or on n of them that another object owns at ptr."""
    return torch.as_tensor(_Array(buffer, buffer.ptr if ptr is None else ptr, buffer.n if n is None else n), device="cuda")


def make_mesh(c, seed):
    el = c["el"]
    pert = 0.0 if c["affine"] else 0.1
    return bp.Mesh(c["nx"], c["ny"], c["nz"], N=c["N"], affine=c["affine"], Nfields=fields(c["bp"], el), pert=pert,
                   pert_seed=1 + seed, dim=3 if el in ("hex", "tet") else 2, simplex=el in ("tri", "tet"))


def make_vector(n, seed):
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1


def prepare(c, seed):
    seed = int(seed) % (1 << 30)
    s = {"case": c}
    if c["kind"] == "batch":
        probs = [{"nx": c["nx"], "ny": c["ny"], "nz": c["nz"], "N": c["N"], "affine": c["affine"],
                  "pert": 0.0 if c["affine"] else 0.1, "pert_seed": 1 + seed, "nrhs": 4, "rhs_seed": seed}]
        s["batch"] = bp.Batch(probs, bp=c["bp"], lam=LAMBDA, precon="JACOBI", precision="MIXED")
        s["x"] = []
        for k in range(4):
            xp, bq = bp.ctypes.c_void_p(), bp.ctypes.c_void_p()
            bp._check(bp.lib().bp_batch_vectors(s["batch"]._h, k, bp.ctypes.byref(xp), bp.ctypes.byref(bq)))
            s["x"].append(view(s["batch"], s["batch"].Ngather[k], xp.value))
        bp.finish()
        return s
    m = s["mesh"] = make_mesh(c, seed)
    if c["kind"] == "ax" or c["kind"] == "operator":
        s["q"] = bp.DeviceBuffer(m.Ngather)
        view(s["q"]).copy_(make_vector(m.Ngather, seed))
        n = m.NL if c["kind"] == "ax" else m.Ngather
        s["Aq"] = bp.DeviceBuffer(n)
        s["out"] = view(s["Aq"])
        if c["bp"] <= 4:
            m.cubature()
        if c["kind"] == "operator":
            s["problem"] = bp.BP(m, bp=c["bp"], lam=LAMBDA)
    else:
        S = s["problem"] = bp.BP(m, bp=c["bp"], lam=LAMBDA, precon="JACOBI", precision="FP64" if c["kind"] == "cg" else "MIXED")
        s["b"] = S.rhs("RANDOM", seed)
        if c["kind"] == "cg":
            s["x"], s["r"] = bp.DeviceBuffer(S.N), bp.DeviceBuffer(S.N)
            s["out"] = [view(s["x"]), view(s["r"])]
        else:
            s["hb"], s["hx"] = (torch.empty(S.N, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2))
            s["hb"][:] = s["b"].download()
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "ax":
        m, q, Aq = s["mesh"], s["q"], s["Aq"]
        if c["el"] == "tet":
            bp.ax_tet3d(m, q, Aq, LAMBDA)
        elif c["el"] == "tri":
            bp.ax_tri2d(m, q, Aq, LAMBDA)
        elif c["bp"] >= 5:
            bp.ax_hex3d(m, q, Aq, LAMBDA)
        else:
            bp.ax_cub_hex3d(m, c["bp"], q, Aq, LAMBDA)
        return s["out"]
    if c["kind"] == "operator":
        s["problem"].operator(s["q"], s["Aq"])
        return s["out"]
    if c["kind"] == "cg":
        s["x"].zero()
        bp._check(bp.lib().bp_memcpy_dtod(s["r"].ptr, s["b"].ptr, s["b"].nbytes, None))
        st, rnorm, alpha = s["problem"].solve(s["x"], s["r"], tol=0.0, maxit=100)
        return {"x": s["out"][0], "r": s["out"][1], "rnorm": rnorm}
    if c["kind"] == "solve":
        s["problem"].solve_host(s["hb"], s["hx"], tol=TOL, maxit=20000)
        return s["hx"]
    s["batch"].solve(tol=TOL, maxit=20000)
    return s["x"]


# ---------------------------------------------------------------------------
# the same results in plain torch, FP64, from the mesh's arrays
# ---------------------------------------------------------------------------
class Exact:
    """The operators of a case in plain torch on the mesh's own arrays."""

    def __init__(self, c, mesh):
        self.c, self.m, E = c, mesh, mesh.E
        get = lambda name: torch.from_numpy(mesh.array(name)).cuda()   # noqa: E731
        self.map = get("GlobalToLocal").long()
        self.live = self.map >= 0
        self.rows = self.map[self.live]
        el, Nq, b = c["el"], mesh.Nq, c["bp"]
        if el in ("tri", "tet"):
            k = 3 if el == "tri" else 6
            self.S = get("S").view(k, mesh.Np, mesh.Np)
            self.MM = get("MM").view(mesh.Np, mesh.Np)
            self.g, self.w = get("ggeo").view(E, k), get("wJ")
            return
        self.curved = not c["affine"]
        if b >= 5:
            self.D, self.T = get("D").view(Nq, Nq), None
            n, names = Nq, ("ggeo", "wJ")
            if c["affine"]:
                gw = get("gllw")
        else:
            n = mesh.cubature().cubNq if self.curved else Nq
            names = ("cubggeo", "cubwJ") if self.curved else ("ggeo", "wJ")
            if self.curved:
                self.T = get("cubInterp").view(n, Nq)
            else:
                self.T = get("invV").view(n, Nq) if b >= 3 else get("MM").view(n, Nq).T.contiguous()
            self.D = get("cubD").view(n, n) if b >= 3 else None
            gw = None
        self.n = n
        dim = 2 if el == "quad" else 3
        ng = 3 if dim == 2 else 6
        pts = n ** dim if self.curved else 1
        G, W = get(names[0]).view(E, pts, ng), get(names[1]).view(E, pts)
        if b >= 5 and c["affine"]:   # the GLL weights
            w = gw
            for _ in range(dim - 1):
                w = (w[:, None] * gw[None, :]).reshape(-1)
            G, W = G * w[None, :, None], W * w[None, :]
        shape = (E,) + ((n,) * dim if G.shape[1] > 1 else (1,) * dim)
        self.G = [G[:, :, a].reshape(shape) for a in range(ng)]
        self.W = W.reshape(shape)

    @staticmethod
    def along(A, u, axis):
        """sum_i A[o, i] u[.., i, ..] along an axis of [E, (k,) j, i]."""
        return torch.movedim(torch.matmul(torch.movedim(u, axis, -1), A.T), -1, axis)

    def field(self, u):
        c, D, T, axes = self.c, self.D, self.T, range(1, u.dim())
        if T is not None:
            for a in axes:
                u = self.along(T, u, a)
        if c["bp"] <= 2:
            r = self.W * u
            if c["affine"]:
                return r
        else:
            d = [self.along(D, u, a) for a in reversed(axes)]     # r, s (, t): the last axis is r
            if len(d) == 2:
                k = ((0, 1), (1, 2))
            else:
                k = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
            r = LAMBDA * self.W * u
            for a, row in zip(reversed(axes), k):
                f = sum(self.G[g] * x for g, x in zip(row, d))
                r = r + self.along(D.T, f, a)
        if T is not None:
            for a in axes:
                r = self.along(T.T, r, a)
        return r

    def local(self, q):
        """The element-local result [E, fields, Np] of A_e q[map]."""
        m, c = self.m, self.c
        u = torch.zeros(m.NL, dtype=torch.float64, device="cuda")
        u[self.live] = q[self.rows]
        if c["el"] in ("tri", "tet"):
            u = u.view(m.E, m.Np)
            r = LAMBDA * self.w[:, None] * (u @ self.MM)
            for a in range(self.S.shape[0]):
                r = r + self.g[:, a:a + 1] * (u @ self.S[a])
            return r.reshape(-1)
        nf = fields(c["bp"], c["el"])
        dim = 2 if c["el"] == "quad" else 3
        u = u.view((m.E, nf) + (m.Nq,) * dim)
        return torch.stack([self.field(u[:, f]) for f in range(nf)], 1).reshape(-1)

    def gather(self, v):
        out = torch.zeros(self.m.Ngather, dtype=torch.float64, device="cuda")
        return out.index_add_(0, self.rows, v[self.live])

    def operator(self, q):
        return self.gather(self.local(q))

    def diagonal(self):
        """Assembled diagonal of the collocated (BP5) stiffness."""
        D2 = (self.D * self.D).T
        dd = torch.diagonal(self.D)
        x, y, z = dd[None, None, None, :], dd[None, None, :, None], dd[None, :, None, None]
        n = self.n
        G = [g.expand(self.m.E, n, n, n) for g in self.G]
        d = LAMBDA * self.W + self.along(D2, G[0], 3) + self.along(D2, G[3], 2) + self.along(D2, G[5], 1)
        d = d + 2 * (x * y * G[1] + x * z * G[2] + y * z * G[4])
        return self.gather(d.reshape(-1))

    def cg(self, b, diag, iters=None, tol=None):
        """Jacobi-PCG from zero, a number of iterations or down to tol: x, the residual and its norms."""
        x, r, norms = torch.zeros_like(b), b.clone(), []
        z = r / diag
        p, rz = z.clone(), torch.dot(r, z)
        stop = None if tol is None else tol * float(b.norm())
        for k in range(iters or 40000):
            Ap = self.operator(p)
            a = rz / torch.dot(p, Ap)
            x += a * p
            r -= a * Ap
            norms.append(r.norm())
            if stop is not None and k % 20 == 19 and float(norms[-1]) <= stop:
                break
            z = r / diag
            new = torch.dot(r, z)
            p.mul_(new / rz).add_(z)
            rz = new
        return x, r, torch.stack(norms)


def exact(c, seed):
    seed = int(seed) % (1 << 30)
    m = make_mesh(c, seed)
    X = Exact(c, m)
    if c["kind"] in ("ax", "operator"):
        q = make_vector(m.Ngather, seed)
        return X.local(q) if c["kind"] == "ax" else X.operator(q)
    diag = (X if c["bp"] == 5 else Exact(dict(c, bp=5), m)).diagonal()
    S = bp.BP(m, bp=c["bp"], lam=LAMBDA)
    rhs = [torch.from_numpy(S.rhs("RANDOM", seed + k).download()).cuda() for k in range(4 if c["kind"] == "batch" else 1)]
    if c["kind"] == "cg":
        x, r, norms = X.cg(rhs[0], diag, iters=100)
        return {"x": x, "r": r, "rnorm": norms}
    if m.NL * iterations(c) * len(rhs) > 3e10:
        return None
    out = [X.cg(b, diag, tol=1e-11)[0] for b in rhs]
    return out if c["kind"] == "batch" else out[0].cpu().numpy()
