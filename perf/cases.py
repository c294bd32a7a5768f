"""What a user of this framework has it do, as cases to be timed.

A user's solver holds a state U on the GPU (or on the host, through the drop-in) and asks, once
per Newton step or line-search trial, for the residual and the tangent of a mesh.  The kinds:

  static     residual and tangent of one phys/ge mesh: a Newton step's assembly
  residual   the residual alone: a line-search trial
  transient  residual and tangent of phys/getime with a traction: a Newton step of a time step
  jacobians  FP64 tangent and both history Jacobians of phys/getime: the transient adjoint's step
  adjoint    forward assembly at element log-scales g, then K^T lambda and dR/dg: a gradient's step
  batch      residual and tangent of many uneven meshes in one call each
  newton     a whole device Newton solve (assemblies, multigrid Krylov solves, line search)
  host       residual and tangent through host pointers (pinned), as the PETSc drop-in calls them

Sizes are elements per direction of quadratic C1 meshes on the unit cube.
"""
import math

import numpy as np
import torch

import igap4standard_b200 as m

DT = 1e-3          # time step of the transient workload
AMP = 1e-3         # seeded-uniform dofs of an assembly check


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the 8^3 configuration: launches and latency decide
        dict(name="static fp64 8^3", kind="static", nx=8, ny=8, nz=8, prec="fp64", perturb=0.0),
        # an ordinary mesh, uneven and with odd sizes, FP32 tangent (inexact Newton)
        dict(name="static fp32 19x26x15", kind="static", nx=19, ny=26, nz=15, prec="fp32", perturb=0.1),
        # the 64^3 configuration, plain FP64 and with the FP32 tangent
        dict(name="static fp64 64^3", kind="static", nx=64, ny=64, nz=64, prec="fp64", perturb=0.1),
        dict(name="static fp32 64^3", kind="static", nx=64, ny=64, nz=64, prec="fp32", perturb=0.1),
        # a line-search trial on a ragged mesh
        dict(name="residual 47x33x52", kind="residual", nx=47, ny=33, nz=52, prec="fp64", perturb=0.1),
        # the 32^3 transient configuration: FP32 tangent, FP64 residual
        dict(name="transient fp32 32^3", kind="transient", nx=32, ny=32, nz=32, prec="fp32", perturb=0.0),
        # one backward step of the transient adjoint on a ragged mesh
        dict(name="jacobians 17x14x11", kind="jacobians", nx=17, ny=14, nz=11, prec="fp64", perturb=0.1),
        # the 32^3 adjoint configuration
        dict(name="adjoint 32^3", kind="adjoint", nx=32, ny=32, nz=32, prec="fp64", perturb=0.0),
        # instances of 6..24 elements per side, as the batched configuration draws them
        dict(name="batch fp32 64", kind="batch", n=64, nmin=6, nmax=24, prec="fp32"),
        dict(name="batch fp64 12", kind="batch", n=12, nmin=6, nmax=24, prec="fp64"),
        # a whole solve: what an application waits for
        dict(name="newton fp32+polish 16^3", kind="newton", nx=16, ny=16, nz=16, prec="fp32", perturb=0.1),
        # the drop-in's host-pointer path: U in, R and all CSR values out
        dict(name="host fp64 24x21x26", kind="host", nx=24, ny=21, nz=26, prec="fp64", perturb=0.1),
    ]


def draw(rng):
    kind = rng.choice(["static", "static", "residual", "transient", "jacobians", "adjoint", "batch", "newton", "host"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "batch":
        nmin = rng.randint(4, 10)
        return dict(kind="batch", n=int(round(math.exp(rng.uniform(math.log(4), math.log(48))))), nmin=nmin,
                    nmax=rng.randint(nmin + 2, 24), prec=prec)
    top = {"static": 60, "residual": 60, "transient": 32, "jacobians": 22, "adjoint": 36, "newton": 18, "host": 30}[kind]
    low = 8 if kind == "newton" else 4
    side = [int(round(math.exp(rng.uniform(math.log(low), math.log(top))))) for _ in range(3)]
    if kind == "newton":       # even, so that the mesh has coarser levels, and nearly cubic
        n = 2 * (side[0] // 2)
        side = [n, n + 2 * rng.randint(-1, 1), n]
    if kind in ("residual", "jacobians", "adjoint"):
        prec = "fp64"
    return dict(kind=kind, nx=side[0], ny=side[1], nz=side[2], prec=prec, perturb=rng.choice([0.0, 0.1, 0.2]))


# ------------------------------------------------------------------ inputs
def _mesh(case, seed):
    ne = (case["nx"], case["ny"], case["nz"])
    return ne, m.knots_for(ne, perturb=case["perturb"], seed=seed)


def _material(case):
    pm = m.par_mat_from_lame(1.0, 1.0, 0.1)
    if case["kind"] in ("transient", "jacobians"):
        pm[5], pm[6], pm[7] = 1.0, 1.0, DT
    return pm


def _vectors(case, seed, count, n):
    """count vectors of n seeded-uniform values in [-1, 1] (float64, on the GPU)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return [torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2.0 - 1.0 for _ in range(count)]


def _states(case, seed, n):
    """(U, U at t_n, U at t_{n-1}): a step's three levels lie near one another."""
    a, b, c = _vectors(case, seed, 3, n)
    u0 = AMP * a
    u1 = u0 + 0.3 * AMP * b
    return u1 + 0.3 * AMP * c, u1, u0


def _instances(case, seed):
    """The batched configuration's meshes (sizes fixed by the case), materials of the seed."""
    inst = m.mesh.batch_config3(n_instances=case["n"], nmin=case["nmin"], nmax=case["nmax"])
    rng = np.random.default_rng(int(seed))
    for c in inst:
        lam, mu = np.exp(rng.normal(0.0, 0.25, 2))
        c["par_mat"] = m.par_mat_from_lame(lam, mu, rng.uniform(0.05, 0.2))
    return inst


def _traction(meta):
    """The transient workload's traction: x direction on the face x = 1."""
    h = np.zeros(len(meta))
    h[(meta[:, 0] == 1) & (meta[:, 1] == 0) & (meta[:, 2] == 0)] = 0.01 * math.sin(2.0 * math.pi * 0.1)
    return h


def prepare(case, seed):
    kind, prec = case["kind"], case["prec"]
    fdt = torch.float64 if prec == "fp64" else torch.float32
    s = dict(kind=kind, prec=prec)
    if kind == "batch":
        A = m.Batch(_instances(case, seed))
        s["U"] = AMP * _vectors(case, seed, 1, A.ndof)[0]
    else:
        ne, kn = _mesh(case, seed)
        phys = "getime" if kind in ("transient", "jacobians") else "ge"
        bc, pd = m.mesh.bc_transient() if phys == "getime" else m.bc_config0()
        A = m.Assembly(ne, kn, _material(case), bc, pd, phys=phys)
        if phys == "getime":
            s["U"], u1, u0 = _states(case, seed, A.ndof)
            torch.cuda.synchronize()
            A.set_history_device(1, u1.data_ptr())
            A.set_history_device(2, u0.data_ptr())
            A.set_neumann_values(_traction(A.neumann_points()[1]))
        else:
            s["U"] = AMP * _vectors(case, seed, 1, A.ndof)[0]
        if kind == "adjoint":
            a, b = _vectors(case, seed + 1, 2, max(A.ndof, A.nelem_total))
            s["lam"], s["g"] = a[:A.ndof].clone(), 0.3 * b[:A.nelem_total].clone()
            s["KT"], s["grad"] = torch.empty_like(s["lam"]), torch.empty_like(s["g"])
        if kind == "newton":
            F0 = np.zeros(9)
            F0[0] = 0.01
            U0 = A.affine_start(kn, F0)
            s["U0"] = torch.as_tensor(U0).cuda() + 0.02 * _free(A) * s["U"]
            s["stream"] = torch.cuda.Stream()
            A.set_stream(s["stream"].cuda_stream)
    s["A"] = A
    if kind == "host":
        s["Uh"] = s.pop("U").cpu().pin_memory().numpy()
        s["Rh"] = torch.empty(A.ndof, dtype=torch.float64).pin_memory().numpy()
        s["Vh"] = torch.empty(A.nnz, dtype=fdt).pin_memory().numpy()
    else:
        s["R"] = torch.empty(A.ndof, dtype=torch.float64, device="cuda")
        if kind not in ("residual", "newton"):
            s["V"] = torch.empty(A.nnz, dtype=fdt, device="cuda")
        if kind == "jacobians":
            s["J1"], s["J0"] = torch.empty_like(s["V"]), torch.empty_like(s["V"])
    torch.cuda.synchronize()
    return s


def _free(A):
    """1 on the dofs without a Dirichlet condition, 0 on the others."""
    f = np.ones(A.ndof)
    f[A.dirichlet_rows()] = 0.0
    return torch.as_tensor(f).cuda()


# ------------------------------------------------------------------ one pass
def run(s):
    A, kind, prec = s["A"], s["kind"], s["prec"]
    if kind == "host":
        return [A.residual(s["Uh"], out=s["Rh"]), A.tangent(s["Uh"], prec, out=s["Vh"])]
    U = s["U"].data_ptr()
    if kind == "residual":
        A.residual_device(U, s["R"].data_ptr())
        return [s["R"]]
    if kind in ("static", "transient", "batch"):
        A.residual_device(U, s["R"].data_ptr())
        A.tangent_device(U, s["V"].data_ptr(), prec)
        return [s["R"], s["V"]]
    if kind == "jacobians":
        A.tangent_device(U, s["V"].data_ptr(), prec)
        A.history_jacobian_device(U, s["J1"].data_ptr(), 1, prec)
        A.history_jacobian_device(U, s["J0"].data_ptr(), 2, prec)
        return [s["V"], s["J1"], s["J0"]]
    if kind == "adjoint":
        A.adjoint_forward_device(s["g"].data_ptr(), U, s["R"].data_ptr(), s["V"].data_ptr(), prec)
        A.adjoint_backward_device(U, s["V"].data_ptr(), s["lam"].data_ptr(), s["KT"].data_ptr(), s["grad"].data_ptr(),
                                  prec)
        return [s["R"], s["V"], s["KT"], s["grad"]]
    with torch.cuda.stream(s["stream"]):
        s["U"].copy_(s["U0"])
    A.newton_solve_device(U, prec, ksp_rtol=1e-10, fp64_polish=prec == "fp32")
    return [s["U"]]


# ------------------------------------------------------------------ what a pass cannot do without
# Operations per element.  The field at the 64 Gauss points and its transpose, by sum factorisation;
# the point integrand (758: the reference's residual integrand); the tangent's contraction of the
# 27 x 27 point matrices, by sum factorisation over 3 full and 3 symmetric component pairs.
_FIELD = 2 * (972 * 3 + 864 * 3 + 64 * 30 * 3)
_RES = 2 * _FIELD + 64 * 758
_TAN = _FIELD + 64 * 2 * 378 * 4 + 2 * (3 * (81 * 576 + 36 * 1296 + 9 * 2916) + 3 * (45 * 576 + 21 * 1296 + 6 * 2916))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = [c["nelem"] for c in _instances(case, 3)]
    else:
        sizes = [(case["nx"], case["ny"], case["nz"])]
    nel = sum(a * b * c for a, b, c in sizes)
    ndof = sum(m.n_dof(s) for s in sizes)
    nnz = sum(m.nnz_of(s) for s in sizes)
    v = 8 if case["prec"] == "fp64" else 4
    lev = 3 if kind in ("transient", "jacobians") else 1
    res = dict(bytes=8 * ndof * (lev + 1), flops=nel * (_RES + (lev - 1) * _FIELD))
    tan = dict(bytes=8 * ndof * lev + v * nnz, flops=nel * (_TAN + (lev - 1) * _FIELD))
    if kind == "residual":
        return res
    if kind == "jacobians":
        return dict(bytes=3 * tan["bytes"], flops=3 * tan["flops"])
    b, f = res["bytes"] + tan["bytes"], res["flops"] + tan["flops"]
    if kind == "adjoint":     # K^T lambda reads the values once more; dR/dg is a residual-like pass
        b += v * nnz + 16 * ndof + 16 * nel
        f += 2 * nnz + res["flops"]
    if kind == "newton":      # five steps, each some 12 products with the tangent
        b, f = 5 * (b + 12 * v * nnz), 5 * (f + 24 * nnz)
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ the same in plain torch, 64 bits
_GX = np.polynomial.legendre.leggauss(4)
_KX, _KY, _KZ = (0, 1, 0, 0, 2, 1, 1, 0, 0, 0), (0, 0, 1, 0, 0, 1, 0, 2, 1, 0), (0, 0, 0, 1, 0, 0, 1, 0, 1, 2)
_I6 = ((0, 1, 2), (1, 3, 4), (2, 4, 5))


def _basis(kv, n):
    """[n, 4, 3 functions, 3 derivatives] of the open quadratic B-splines, weights [n, 4]."""
    kv = np.asarray(kv, dtype=np.float64)
    lo, hi = kv[2:2 + n, None], kv[3:3 + n, None]
    x = lo + (hi - lo) * (0.5 + 0.5 * _GX[0])
    w = (hi - lo) * 0.5 * _GX[1]
    a, b, c, d = (kv[k:k + n, None] for k in (1, 2, 3, 4))
    p, q, h = c - a, d - b, c - b
    one = np.ones_like(x)
    n0 = [(c - x) ** 2 / (p * h), -2 * (c - x) / (p * h), 2 / (p * h) * one]
    n2 = [(x - b) ** 2 / (q * h), 2 * (x - b) / (q * h), 2 / (q * h) * one]
    n1 = [(x - a) * (c - x) / (p * h) + (d - x) * (x - b) / (q * h),
          (c + a - 2 * x) / (p * h) + (d + b - 2 * x) / (q * h), -2 / (p * h) * one - 2 / (q * h) * one]
    t = np.stack([np.stack(f, -1) for f in (n0, n1, n2)], axis=2)
    return torch.as_tensor(t).cuda(), torch.as_tensor(w).cuda()


class _Plain:
    """Residual and tangent of one mesh in plain torch, FP64, element blocks at a time."""

    def __init__(self, ne, knots, par):
        self.ne, self.nb = ne, tuple(n + 2 for n in ne)
        off, self.tab, self.kv = 0, [], []
        for n in ne:
            self.kv.append(np.asarray(knots[off:off + n + 5]))
            self.tab.append(_basis(self.kv[-1], n))
            off += n + 5
        self.par = par
        self.nel, self.ndof = int(np.prod(ne)), 3 * int(np.prod(self.nb))
        lo = [np.maximum(np.arange(b) - 2, 0) for b in self.nb]
        width = [np.minimum(np.arange(b) + 2, b - 1) - l + 1 for b, l in zip(self.nb, lo)]
        self.lo, self.width = ([torch.as_tensor(v).cuda() for v in w] for w in (lo, width))
        per = (width[0][:, None, None] * width[1][None, :, None] * width[2][None, None, :]).reshape(-1) * 3
        self.rowptr = torch.as_tensor(np.concatenate([[0], np.cumsum(np.repeat(per, 3))])).cuda()
        self.nnz = int(self.rowptr[-1])

    def blocks(self, size):
        for i in range(0, self.nel, size):
            e = torch.arange(i, min(i + size, self.nel), device="cuda")
            ez, ey, ex = e % self.ne[2], (e // self.ne[2]) % self.ne[1], e // (self.ne[1] * self.ne[2])
            o = torch.arange(3, device="cuda")
            cx, cy, cz = ex[:, None] + o, ey[:, None] + o, ez[:, None] + o
            cp = ((cx[:, :, None, None] * self.nb[1] + cy[:, None, :, None]) * self.nb[2] + cz[:, None, None, :])
            (tx, wx), (ty, wy), (tz, wz) = self.tab
            tx, ty, tz = tx[ex], ty[ey], tz[ez]
            # N[e, q, derivative, a], q = (x, y, z)
            N = torch.stack([torch.einsum("eqa,erb,esc->eqrsabc", tx[..., _KX[k]], ty[..., _KY[k]], tz[..., _KZ[k]])
                             .reshape(len(e), 64, 27) for k in range(10)], dim=2)
            w = torch.einsum("eq,er,es->eqrs", wx[ex], wy[ey], wz[ez]).reshape(len(e), 64)
            yield e, (cx, cy, cz), cp.reshape(len(e), 27), N, w

    def field(self, U, cp, N):
        """[e, q, 3 components, 10 derivatives]"""
        return torch.einsum("eqka,eai->eqik", N, U.reshape(-1, 3)[cp])

    # strains e = (E00, E11, E22, E01, E02, E12, E_II,K at 6 + 3 I + K); W = Phi(e)
    def strains(self, u):
        F = u[..., 1:4] + torch.eye(3, dtype=torch.float64, device="cuda")
        G = u[..., 4:10]
        C = 0.5 * torch.einsum("eqki,eqkj->eqij", F, F)
        E = [C[..., 0, 0] - 0.5, C[..., 1, 1] - 0.5, C[..., 2, 2] - 0.5, C[..., 0, 1], C[..., 0, 2], C[..., 1, 2]]
        for I in range(3):
            for K in range(3):
                E.append((F[..., I] * G[..., _I6[I][K]]).sum(-1))
        return F, G, torch.stack(E, -1)

    def energy(self, E, second):
        r, cu, p2, p3 = self.par[:4]
        f = 4.0 / 3.0 * r * (1.0 - cu)
        den = r * r * (1.0 - 2.0 * cu) - r * f
        c36, c37, c38, p4 = -f / (r * r * den), 2.0 * cu / den, -1.0 / (r * r * den), self.par[4] ** 2
        q2, q3, q6 = 2.0 ** -0.5, 3.0 ** -0.5, 6.0 ** -0.5
        T = torch.zeros(12, 15, dtype=torch.float64, device="cuda")     # v = T e
        T[0, 0] = T[0, 1] = T[0, 2] = q3
        T[1, 0], T[1, 1] = q2, -q2
        T[2, 0], T[2, 1], T[2, 2] = q6, q6, -2 * q6
        T[3, 3] = T[4, 4] = T[5, 5] = 1.0
        for K in range(3):
            T[6 + K, 6 + K], T[6 + K, 9 + K] = q2, -q2
            T[9 + K, 6 + K], T[9 + K, 9 + K], T[9 + K, 12 + K] = q6, q6, -2 * q6
        v = E @ T.T
        k = torch.tensor([2 * p2, 0, 0] + [2 * p3] * 3 + [2 * p4] * 6, dtype=torch.float64, device="cuda")
        d = v * k
        a, b = v[..., 1], v[..., 2]
        s2 = a * a + b * b
        d[..., 1] = -6 * c36 * a * b + 2 * c37 * a + 4 * c38 * s2 * a
        d[..., 2] = 3 * c36 * (b * b - a * a) + 2 * c37 * b + 4 * c38 * s2 * b
        if not second:
            return d @ T, None
        H = torch.diag(k).expand(v.shape[:-1] + (12, 12)).clone()
        H[..., 1, 1] = -6 * c36 * b + 2 * c37 + 4 * c38 * (3 * a * a + b * b)
        H[..., 2, 2] = 6 * c36 * b + 2 * c37 + 4 * c38 * (a * a + 3 * b * b)
        H[..., 1, 2] = H[..., 2, 1] = -6 * c36 * a + 8 * c38 * a * b
        return d @ T, T.T @ H @ T

    def bmat(self, F, G):
        """d strains / d (component, derivative 1..9): [e, q, 15, 3, 9]"""
        B = torch.zeros(F.shape[:2] + (15, 3, 9), dtype=torch.float64, device="cuda")
        for r, (I, J) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            B[..., r, :, I] += 0.5 * F[..., J]
            B[..., r, :, J] += 0.5 * F[..., I]
        for I in range(3):
            for K in range(3):
                B[..., 6 + 3 * I + K, :, I] += G[..., _I6[I][K]]
                B[..., 6 + 3 * I + K, :, 3 + _I6[I][K]] += F[..., I]
        return B

    def gradient(self, u):
        """dW/d(component, derivative): [e, q, 3, 10]"""
        F, G, E = self.strains(u)
        d, _ = self.energy(E, False)
        r = torch.zeros_like(u)
        r[..., 1:] = torch.einsum("eqs,eqskm->eqkm", d, self.bmat(F, G))
        return r

    def hessian(self, u):
        """d2W on the derivatives 1..9: [e, q, 3, 9, 3, 9]"""
        F, G, E = self.strains(u)
        d, H = self.energy(E, True)
        B = self.bmat(F, G).flatten(-2)
        D = (B.transpose(-1, -2) @ (H @ B)).unflatten(-1, (3, 9)).unflatten(-3, (3, 9))
        geo = torch.zeros(d.shape[:2] + (9, 9), dtype=torch.float64, device="cuda")
        for r, (I, J) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            geo[..., I, J] += 0.5 * d[..., r]
            geo[..., J, I] += 0.5 * d[..., r]
        for I in range(3):
            for K in range(3):
                geo[..., I, 3 + _I6[I][K]] += d[..., 6 + 3 * I + K]
                geo[..., 3 + _I6[I][K], I] += d[..., 6 + 3 * I + K]
        for k in range(3):
            D[..., k, :, k, :] += geo
        return D

    @staticmethod
    def taylor(c, degree):
        """Nodes s_j and weights with sum_j weight_j f(s_j) = sum_n c_n (coefficient n of f), f of that degree."""
        s = np.cos((np.arange(degree + 1) + 0.5) * math.pi / (degree + 1))
        V = np.vander(s, degree + 1, increasing=True).astype(np.float64)
        rhs = np.zeros(degree + 1)
        rhs[:len(c)] = c
        return s, np.linalg.solve(V.T, rhs)

    def integrand(self, us, what):
        """The point residual [e, q, 3, 10] ("r"), or the point matrix [e, q, 3, 9, 3, 9] and the coefficient of
        the value components ("k": tangent, "1" / "2": history Jacobians); us: one field, or three levels."""
        if len(us) == 1:
            return self.gradient(us[0]) if what == "r" else (self.hessian(us[0]), 0.0)
        u, u1, u0 = us
        mid, h = 0.5 * (u0 + u1), 0.5 * (u - u0)
        rho, cii, dt = self.par[5:8]
        if what == "r":
            r = sum(w * self.gradient(mid + s * h) for s, w in zip(*self.taylor([1, 1 / 2, 1 / 3, 1 / 4], 7)))
            r[..., 0] = cii * (u - u0)[..., 0] / (2 * dt) + rho * (u + u0 - 2 * u1)[..., 0] / (dt * dt)
            return r
        c, mass = {"k": ([1 / 4, 1 / 6, 1 / 8], rho / dt ** 2 + cii / (2 * dt)),
                   "1": ([1 / 2, 1 / 4, 1 / 6, 1 / 8], -2 * rho / dt ** 2),
                   "2": ([1 / 4, 1 / 12, 1 / 24, 1 / 8], rho / dt ** 2 - cii / (2 * dt))}[what]
        return sum(w * self.hessian(mid + s * h) for s, w in zip(*self.taylor(c, 6))), mass

    def residual(self, us, scale=None, lam=None):
        """R, and lam . R_e per element where lam is given."""
        R, grad = torch.zeros(self.ndof, dtype=torch.float64, device="cuda"), []
        for e, _, cp, N, w in self.blocks(2048):
            r = self.integrand([self.field(u, cp, N) for u in us], "r")
            w = w if scale is None else w * scale[e][:, None]
            Re = torch.einsum("eq,eqik,eqka->eai", w, r, N)
            R.view(-1, 3).index_add_(0, cp.reshape(-1), Re.reshape(-1, 3))
            if lam is not None:
                grad.append((Re * lam.view(-1, 3)[cp]).sum((1, 2)))
        return R, torch.cat(grad) if grad else None

    def tangent(self, us, what="k", scale=None):
        V = torch.zeros(self.nnz, dtype=torch.float64, device="cuda")
        k3 = torch.arange(3, device="cuda")
        for e, (cx, cy, cz), cp, N, w in self.blocks(512 if len(us) == 3 else 1024):
            D, mass = self.integrand([self.field(u, cp, N) for u in us], what)
            w = w if scale is None else w * scale[e][:, None]
            n = len(e)
            M = N[:, :, 1:]                                                             # [e, q, 9, 27]
            T = (D.reshape(n, 64, 81, 9) @ M) * w[:, :, None, None]                      # [e, q, (k m l), b]
            T = T.view(n, 64, 3, 9, 81).permute(0, 1, 3, 2, 4).reshape(n, 576, 243)      # [(q m), (k l b)]
            K = (M.reshape(n, 576, 27).transpose(1, 2) @ T).view(n, 27, 3, 3, 27).permute(0, 1, 2, 4, 3).clone()
            if mass:
                B = torch.einsum("eqa,eq,eqb->eab", N[:, :, 0], w, N[:, :, 0]) * mass
                for k in range(3):
                    K[:, :, k, :, k] += B
            # position of entry (a, k; b, l) in its CSR row
            def at(c, d):
                return c[:, None, :] - self.lo[d][c][:, :, None]                         # [e, row, column]
            px, py, pz = at(cx, 0), at(cy, 1), at(cz, 2)
            wy, wz = self.width[1][cy], self.width[2][cz]
            pos = (px[:, :, None, None, :, None, None] * wy[:, None, :, None, None, None, None]
                   + py[:, None, :, None, None, :, None]) * wz[:, None, None, :, None, None, None] \
                + pz[:, None, None, :, None, None, :]
            pos = pos.reshape(n, 27, 1, 27, 1) * 3 + k3
            pos = pos + self.rowptr[3 * cp[:, :, None] + k3][:, :, :, None, None]
            V.index_add_(0, pos.reshape(-1), K.reshape(-1))
        return V

    def rows(self):
        return torch.repeat_interleave(torch.arange(self.ndof, device="cuda"), self.rowptr[1:] - self.rowptr[:-1])

    def columns(self):
        r = self.rows()
        p = torch.arange(self.nnz, device="cuda") - self.rowptr[r]
        cp = r // 3
        z, y, x = cp % self.nb[2], (cp // self.nb[2]) % self.nb[1], cp // (self.nb[1] * self.nb[2])
        k, p = p % 3, p // 3
        wz, wy = self.width[2][z], self.width[1][y]
        cz, p = p % wz + self.lo[2][z], p // wz
        cy, cx = p % wy + self.lo[1][y], p // wy + self.lo[0][x]
        return 3 * ((cx * self.nb[1] + cy) * self.nb[2] + cz) + k

    def affine(self, F0):
        g = [torch.as_tensor(0.5 * (k[1:-2] + k[2:-1])).cuda() for k in self.kv]
        X = torch.stack(torch.meshgrid(*g, indexing="ij"), -1).reshape(-1, 3)
        return (X @ torch.as_tensor(np.asarray(F0, dtype=np.float64).reshape(3, 3)).cuda().T).reshape(-1)

    def dirichlet(self, transient):
        """(mask of the Dirichlet dofs, their values): x = 0 clamped in value and slope (the first two layers
        of control points), and for the static problems u_x = 0.01 on x = 1."""
        f = torch.zeros(self.nb[0], self.nb[1] * self.nb[2], 3, dtype=torch.bool, device="cuda")
        g = torch.zeros(f.shape, dtype=torch.float64, device="cuda")
        f[0:2] = True
        if not transient:
            f[-1, :, 0] = True
            g[-1, :, 0] = 0.01
        return f.reshape(-1), g.reshape(-1)

    def traction(self):
        """Surface term of the constant x traction on x = 1."""
        b = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in self.nb]
        for d in (1, 2):
            t, w = self.tab[d]
            for a in range(3):
                b[d][a:a + self.ne[d]] += (t[:, :, a, 0] * w).sum(1)
        R = torch.zeros(self.nb + (3,), dtype=torch.float64, device="cuda")
        R[-1, :, :, 0] = b[1][:, None] * b[2][None, :] * (0.01 * math.sin(2.0 * math.pi * 0.1))
        return R.reshape(-1)

    def with_rows(self, R, us, transient):
        f, g = self.dirichlet(transient)
        return torch.where(f, us[0] - g, R)

    def eliminated(self, V, transient, columns=True):
        f, _ = self.dirichlet(transient)
        r = self.rows()
        if not columns:
            return V.masked_fill_(f[r], 0.0)
        c = self.columns()
        V.masked_fill_(f[r] | f[c], 0.0)
        return V.masked_fill_((r == c) & f[r], 1.0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        inst = _instances(case, seed)
        U = AMP * _vectors(case, seed, 1, sum(m.n_dof(c["nelem"]) for c in inst))[0]
        R, V, o = [], [], 0
        for c in inst:
            P = _Plain(c["nelem"], c["knots"], c["par_mat"])
            u = [U[o:o + P.ndof]]
            o += P.ndof
            R.append(P.with_rows(P.residual(u)[0], u, False))
            V.append(P.eliminated(P.tangent(u), False))
        return [torch.cat(R), torch.cat(V)]
    ne, kn = _mesh(case, seed)
    P = _Plain(ne, kn, _material(case))
    if kind in ("transient", "jacobians"):
        us = list(_states(case, seed, P.ndof))
        if kind == "jacobians":
            return [P.eliminated(P.tangent(us), True), P.eliminated(P.tangent(us, "1"), True, columns=False),
                    P.eliminated(P.tangent(us, "2"), True, columns=False)]
        return [P.with_rows(P.residual(us)[0] - P.traction(), us, True), P.eliminated(P.tangent(us), True)]
    us = [AMP * _vectors(case, seed, 1, P.ndof)[0]]
    if kind == "newton":
        return _newton(P, us[0])
    if kind == "adjoint":
        a, b = _vectors(case, seed + 1, 2, max(P.ndof, P.nel))
        lam, scale = a[:P.ndof], torch.exp(0.3 * b[:P.nel])
        f, _ = P.dirichlet(False)
        R, grad = P.residual(us, scale, torch.where(f, 0.0, lam))
        V = P.eliminated(P.tangent(us, scale=scale), False)
        KT = torch.zeros_like(lam).index_add_(0, P.columns(), V * lam[P.rows()])
        return [P.with_rows(R, us, False), V, KT, grad]
    R = P.with_rows(P.residual(us)[0], us, False)
    return [R] if kind == "residual" else [R, P.eliminated(P.tangent(us), False)]


def _newton(P, u):
    """The solution by full Newton steps with a dense factorisation; None where that is too large."""
    if P.ndof > 20000:
        return None
    f, g = P.dirichlet(False)
    U = torch.where(f, g, P.affine([0.01, 0, 0, 0, 0, 0, 0, 0, 0]) + 0.02 * u)
    for _ in range(8):
        R = P.with_rows(P.residual([U])[0], [U], False)
        V = P.eliminated(P.tangent([U]), False)
        K = torch.zeros(P.ndof, P.ndof, dtype=torch.float64, device="cuda")
        K[P.rows(), P.columns()] = V
        d = torch.linalg.solve(K, R)
        U = U - d
        if float(d.abs().max()) < 1e-15:
            break
    return [U]
