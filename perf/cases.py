"""Workloads that are timed and compared when a kernel changes.

`listed()` names the standing cases, `draw(rng)` makes one more of the same ranges, `prepare`
builds what a program holds before the call (mesh, handle, fields on the GPU), `run` makes the
call through the package's public entry points, `work` counts what the call cannot do without,
and `exact` evaluates the same operators in 64 bits with plain torch: dense 1D contractions on
all quadrature points, every face once, derivatives by torch's autograd, no code of this package.

Kinds of case:
  rhs        the fused explicit right-hand sides of one IMEX stage (the benchmark's apply)
  rhs_split  the same three right-hand sides by the three calls the stage drivers make
  backward   vector-Jacobian product of the fused right-hand sides
  tangent    Jacobian-vector product of the fused right-hand sides
  implicit   the implicit operators of one stage: B, C, A, A^{-1}, M^{-1}, the Schur complement
  solve      set-up of the Schur pressure solver and one solve to a relative residual of 1e-10
  imex       one IMEX step from a given state
  imex_grad  one recorded IMEX step and its adjoint

All meshes are the 2D terrain-following hill (40 km x 16 km, Witch of Agnesi) or the annulus with
radial gravity; fields are the hydrostatic background with seeded smooth perturbations of
relative size 1e-3 and a 10 m/s wind.
"""
import math

import numpy as np
import torch

GAMMA, R_GAS, CP, G_ACC = 1.4, 287.0, 1004.5, 9.81
P_REF = 1.0e5
RHO_REF = P_REF / (R_GAS * 300.0)
MA, FR = math.sqrt(RHO_REF / P_REF), 1.0 / math.sqrt(G_ACC)
G1, GG = 1.0 / (GAMMA - 1.0), GAMMA / (GAMMA - 1.0)
EARTH = 6.37122e6
SPONGE = (10000.0, 16000.0, 0.02, -20000.0, 20000.0, 4000.0, 0.01, 10.0)  # z0, z1, rate, x0, x1, width, rate, u_ref
MODES = 16


# ------------------------------------------------------------------ the cases
def _case(name, kind, nx, nz, degree, **more):
    c = {"kind": kind, "nx": nx, "nz": nz, "degree": degree, "mesh": "hill", "periodic": True, "stage": 1}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the small hill case of a laptop-size study: one launch, all latency; sponge layers on
        _case("rhs_40x16_p4_sponge", "rhs", 40, 16, 4, sponge=True),
        # the benchmark's apply: 13.1 M degrees of freedom, walled hill
        _case("rhs_512x256_p4", "rhs", 512, 256, 4, periodic=False),
        # low order, odd sizes, the stage with two explicit groups, as the stage drivers call it
        _case("rhs_split_501x255_p2_s2", "rhs_split", 501, 255, 2, stage=2, periodic=False),
        # production size: 105 M degrees of freedom, the stage with three explicit groups
        _case("rhs_2048x512_p4_s3", "rhs", 2048, 512, 4, stage=3),
        # the implicit operators one by one, at the highest degree, odd sizes
        _case("implicit_255x127_p6", "implicit", 255, 127, 6, periodic=False, stage=2),
        # gradient of the explicit operator at the benchmark's size
        _case("backward_512x256_p4", "backward", 512, 256, 4),
        # the pressure Helmholtz solve on the hill scaled to 1024x256 cells, FP32 polynomial preconditioner
        _case("solve_cheb32_1024x256_p4", "solve", 1024, 256, 4, precond="cheb_fp32"),
        # the same system by the FP32 multigrid preconditioner at an ordinary size
        _case("solve_mg32_256x128_p3", "solve", 256, 128, 3, precond="mg_fp32"),
        # a step of the small hill case with the default options (FP64, the reference's GMRES criterion)
        _case("imex_40x16_p4", "imex", 40, 16, 4, precond="default", eps=1e-8),
        # the benchmark's step, mixed precision
        _case("imex_mixed_512x256_p4", "imex", 512, 256, 4, precond="cheb_fp32", eps=1e-8),
        # its FP64 counterpart (Jacobi) at an ordinary size
        _case("imex_fp64_256x128_p4", "imex", 256, 128, 4, precond="jacobi", eps=1e-8),
        # a step and its adjoint, as a checkpointed gradient repeats them
        _case("imex_grad_128x64_p4", "imex_grad", 128, 64, 4, precond="cheb_fp32", eps=1e-10),
    ]


# scalar nodes that a drawn case of each kind has at most
_MOST = {"rhs": 26e6, "rhs_split": 5e6, "backward": 3.3e6, "tangent": 3.3e6, "implicit": 1.6e6, "solve": 3.3e6,
         "imex": 1.6e6, "imex_grad": 2.1e5}
_LEAST = {"rhs": 3e3, "rhs_split": 3e3, "backward": 3e3, "tangent": 3e3, "implicit": 3e3, "solve": 1.6e4, "imex": 4e3,
          "imex_grad": 4e3}


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "rhs_split", "backward", "tangent", "implicit", "solve", "solve", "imex",
                       "imex", "imex_grad"])
    degree = rng.choice([1, 2, 3, 4, 4, 4, 5, 6] if kind in ("rhs", "rhs_split", "implicit") else [2, 3, 4, 4, 5])
    cells = math.exp(rng.uniform(math.log(_LEAST[kind]), math.log(_MOST[kind]))) / (degree + 1) ** 2
    aspect = math.exp(rng.uniform(math.log(1.2), math.log(5.0)))
    nx, nz = max(4, round(math.sqrt(cells * aspect))), max(3, round(math.sqrt(cells / aspect)))
    if rng.random() < 0.5 or kind == "solve":  # even sizes, as a mesh that was refined has (multigrid needs them)
        nx, nz = nx + nx % 2, nz + nz % 2
    c = _case(None, kind, nx, nz, degree, stage=rng.choice([1, 2, 3]))
    if kind == "solve":
        c.update(stage=rng.choice([1, 2]), precond=rng.choice(["cheb_fp32", "cheb_fp32", "mg_fp32", "cheb_fp64", "jacobi"]))
        if c["precond"] in ("jacobi", "cheb_fp64") and cells * (degree + 1) ** 2 > 8e5:
            c["precond"] = "cheb_fp32"
    elif kind in ("imex", "imex_grad"):
        c.update(stage=1, precond="cheb_fp32", eps=rng.choice([1e-8, 1e-10]) if kind == "imex" else 1e-10)
        if kind == "imex" and rng.random() < 0.4 and cells * (degree + 1) ** 2 < 4e5:
            c.update(precond=rng.choice(["jacobi", "default"]), eps=1e-8)
    elif kind == "implicit":
        c.update(stage=rng.choice([1, 2]), periodic=rng.random() < 0.5)
    elif kind in ("rhs", "rhs_split"):
        if rng.random() < 0.2:
            c.update(mesh="annulus")
        else:
            c.update(periodic=rng.random() < 0.5, sponge=rng.random() < 0.25)
    else:
        c.update(periodic=rng.random() < 0.5)
    return c


def _dt(c):
    """The time step a run of this mesh takes: the acoustic Courant number of the 512x256 hill at 0.5 s."""
    return min(2.0, 0.5 * min(512.0 / c["nx"], 256.0 / c["nz"]) * 4.0 / max(4, c["degree"]))


# ------------------------------------------------------------------ mesh and fields
def _vertices(c):
    """(nz+1, nx+1, 2) float64"""
    nx, nz = c["nx"], c["nz"]
    v = np.empty((nz + 1, nx + 1, 2))
    if c["mesh"] == "annulus":
        th = -2.0 * np.pi * np.arange(nx + 1) / nx
        th[-1] = 0.0
        r = np.linspace(0.9 * EARTH, EARTH, nz + 1)
        v[..., 0] = r[:, None] * np.cos(th)
        v[..., 1] = r[:, None] * np.sin(th)
    else:
        x, zeta = np.linspace(-20000.0, 20000.0, nx + 1), np.linspace(0.0, 16000.0, nz + 1)
        h = 400.0 / (1.0 + (x / 1000.0) ** 2)
        v[..., 0] = x
        v[..., 1] = h + zeta[:, None] * (1.0 - h / 16000.0)
    return v


def _gll(p):
    inner = np.sort(np.real(np.polynomial.legendre.Legendre.basis(p).deriv().roots())) if p > 1 else np.empty(0)
    d1 = np.polynomial.legendre.Legendre.basis(p).deriv()
    for _ in range(4):
        inner = inner - d1(inner) / d1.deriv()(inner) if p > 1 else inner
    return 0.5 * (np.concatenate([[-1.0], inner, [1.0]]) + 1.0)


class _Fields:
    """Seeded smooth fields at the DoF points, on the GPU."""

    def __init__(self, c, seed):
        self.c, self.rng = c, np.random.default_rng(seed)
        self.dev = torch.device("cuda")
        p1 = c["degree"] + 1
        s = _gll(c["degree"])
        x = (np.arange(c["nx"])[:, None] + s).reshape(-1) / c["nx"]
        z = (np.arange(c["nz"])[:, None] + s).reshape(-1) / c["nz"]
        k = np.arange(1, MODES + 1)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        ax, az = 2 * np.pi * np.outer(x, k), np.pi * np.outer(z, k)
        self.cx, self.sx, self.cz, self.sz = t(np.cos(ax)), t(np.sin(ax)), t(np.cos(az)), t(np.sin(az))
        self.shape = (c["nz"], p1, c["nx"], p1)
        self.k2 = k[:, None] ** 2 + k[None, :] ** 2
        if c["mesh"] == "annulus":
            height = t(z * 0.1 * EARTH * 0.16)  # the background up to about 100 km of scaled height stays positive
            height = (height / height.max() * 16000.0)[:, None].expand(-1, x.size)
        else:
            h = np.interp(x * c["nx"], np.arange(c["nx"] + 1), 400.0 / (1.0 + (np.linspace(-20, 20, c["nx"] + 1)) ** 2))
            height = t(h)[None, :] + t(16000.0 * z)[:, None] * (1.0 - t(h)[None, :] / 16000.0)
        n = 0.01
        th = 300.0 * torch.exp(n * n * height / G_ACC)
        ex = 1.0 + G_ACC**2 / (CP * 300.0 * n * n) * (torch.exp(-n * n * height / G_ACC) - 1.0)
        self.p_b = ex ** (CP / R_GAS)
        self.rho_b = self.p_b * P_REF / (R_GAS * th * ex) / RHO_REF

    def _smooth(self, amplitude=1e-3):
        """A field on the node grid with |.| <= amplitude (about)."""
        a = self.rng.standard_normal((MODES, MODES)) / self.k2
        ph, ps = self.rng.uniform(0, 2 * np.pi, (2, MODES, MODES))
        m = lambda w: torch.from_numpy(w.T.copy()).to(self.dev)  # noqa: E731  (l, k)
        f = self.cz @ (m(a * np.cos(ph) * np.cos(ps)) @ self.cx.T - m(a * np.sin(ph) * np.cos(ps)) @ self.sx.T)
        f -= self.sz @ (m(a * np.cos(ph) * np.sin(ps)) @ self.cx.T - m(a * np.sin(ph) * np.sin(ps)) @ self.sx.T)
        return f * (amplitude / f.abs().max())

    def _vec(self, *grids):
        """Node grids -> DoF vector, cell-major, component-blocked."""
        g = torch.stack([x.reshape(self.shape).permute(0, 2, 1, 3) for x in grids], dim=2)
        return g.reshape(-1).contiguous()

    def rho(self):
        return self._vec(self.rho_b * (1.0 + self._smooth()))

    def p(self):
        return self._vec(self.p_b * (1.0 + self._smooth()))

    def u(self):
        return self._vec(10.0 * (1.0 + self._smooth()), 10.0 * self._smooth())

    def any(self, comps, amplitude=1.0):
        return self._vec(*[self._smooth(amplitude) for _ in range(comps)])

    def noise(self, comps):
        g = torch.Generator(device=self.dev)
        g.manual_seed(int(self.rng.integers(1 << 62)))
        n = comps * self.shape[0] * self.shape[1] * self.shape[2] * self.shape[3]
        return torch.randn(n, dtype=torch.float64, device=self.dev, generator=g)

    def sources(self):
        """The source list of the fused right-hand sides of the case's stage."""
        f = []
        for _ in range(self.c["stage"]):
            f += [self.rho(), self.u(), self.p()]
        return f + [self.rho(), self.u()]


def _inputs(c, seed):
    """Everything the call reads, from the seed alone."""
    f, kind = _Fields(c, seed), c["kind"]
    d = {}
    if kind in ("rhs", "rhs_split", "backward", "tangent"):
        d["src"] = f.sources()
        if kind == "backward":  # a functional's gradient: smooth with a rough part
            d["ybar"] = [f.any(1) + 0.1 * f.noise(1), f.any(2) + 0.1 * f.noise(2), f.any(1) + 0.1 * f.noise(1)]
        if kind == "tangent":
            d["dsrc"] = [f.any(s.numel() // d["src"][0].numel(), 1e-3) for s in d["src"]]
    elif kind == "implicit":
        d.update(rho=f.rho(), pf=f.p(), p=f.p(), w=f.u(), v=f.any(2) + 0.1 * f.noise(2), r=f.any(1) + 0.1 * f.noise(1))
    elif kind == "solve":
        d.update(rho=f.rho(), pf=f.p(), b=f.any(1))
    else:
        d.update(rho=f.rho(), u=f.u(), p=f.p())
        if kind == "imex_grad":
            d["ybar"] = [f.any(1), f.any(2), f.any(1)]
    return d


def prepare(case, seed):
    from atmospheric_flows_b200.mesh import Mesh

    c = case
    d = _inputs(c, seed)
    annulus = c["mesh"] == "annulus"
    mesh = Mesh(c["nx"], c["nz"], _vertices(c), bool(annulus or c["periodic"]), 1 if annulus else 0, EARTH if annulus else 0.0)
    s = {"case": c, "in": d}
    if c["kind"] in ("imex", "imex_grad"):
        from atmospheric_flows_b200.imex import IMEXStepper

        more = {} if c["precond"] == "default" else {"schur_preconditioner": c["precond"]}
        s["stepper"] = IMEXStepper(mesh, c["degree"], MA, FR, _dt(c), eps=c["eps"], **more)
        return s
    from atmospheric_flows_b200.operator import EULEROperator

    op = EULEROperator(mesh, c["degree"], MA, FR, _dt(c), stream=torch.cuda.current_stream())
    op.set_HYPERBOLIC_stage(c["stage"])
    if c.get("sponge"):
        op.set_sponge(*SPONGE)
    s["op"] = op
    new = lambda like: torch.empty_like(like)  # noqa: E731
    if c["kind"] in ("rhs", "rhs_split", "tangent"):
        s["out"] = [new(d["src"][0]), new(d["src"][1]), new(d["src"][2])]
    elif c["kind"] == "backward":
        s["out"] = [new(x) for x in d["src"]]
    elif c["kind"] == "implicit":
        op.set_schur_mode(1)
        s["out"] = {"B": new(d["w"]), "C": new(d["p"]), "A": new(d["w"]), "Ainv": new(d["w"]), "Minv": new(d["p"]),
                    "schur": new(d["p"])}
    else:
        from atmospheric_flows_b200.schur import SchurSolver

        op.set_schur_mode(1)
        op.set_rho_for_fixed(d["rho"])
        op.set_pres_fixed(d["pf"])
        s["solver"] = SchurSolver(op, c["precond"])
        s["solver"].setup(estimate_eigenvalues=True)  # once per mesh and time step
        s["x"] = new(d["b"])
    return s


def run(state):
    c, d = state["case"], state["in"]
    kind = c["kind"]
    if kind == "rhs":
        state["op"].vmult_rhs_fused(*state["out"], d["src"])
        return state["out"]
    if kind == "rhs_split":  # the stage drivers' update_density, update_velocity and pressure right-hand sides
        op, s, src = state["op"], c["stage"], d["src"]
        op.vmult_rhs_rho_update(state["out"][0], [x for j in range(s) for x in src[3 * j:3 * j + 2]])
        op.vmult_rhs_velocity_fixed(state["out"][1], src[:3 * s] + (src[3 * s:3 * s + 1] if s < 3 else []))
        op.vmult_rhs_pressure(state["out"][2], src)
        return state["out"]
    if kind == "backward":
        state["op"].vmult_rhs_fused_backward(d["src"], *d["ybar"], state["out"])
        return state["out"]
    if kind == "tangent":
        state["op"].vmult_rhs_fused_tangent(d["src"], d["dsrc"], *state["out"])
        return state["out"]
    if kind == "implicit":  # a new density each time, as each stage of a step sets one
        op, o = state["op"], state["out"]
        op.set_rho_for_fixed(d["rho"])
        op.set_pres_fixed(d["pf"])
        op.vmult_pressure(o["B"], d["p"])
        op.vmult_enthalpy(o["C"], d["w"])
        op.set_NS_stage(3)
        op.vmult(o["A"], d["v"])
        op.vmult_inverse(o["Ainv"], d["v"])
        op.set_NS_stage(1)
        op.vmult_inverse(o["Minv"], d["r"])
        op.set_NS_stage(2)
        op.vmult(o["schur"], d["p"])
        return o
    if kind == "solve":  # a stage's new coefficients, then the solve from zero
        op, x = state["op"], state["x"]
        op.set_rho_for_fixed(d["rho"])
        op.set_pres_fixed(d["pf"])
        state["solver"].setup()
        x.zero_()
        state["solver"].solve(x, d["b"], rel_tol=1e-10, max_iterations=3000)
        return x
    st = state["stepper"]
    if kind == "imex":
        st.set_state(d["rho"], d["u"], d["p"])
        st.step(1)
        return st.get_state()
    y = st.step_forward(d["rho"], d["u"], d["p"])
    return list(y) + list(st.step_backward(*d["ybar"], rel_tol=1e-10))


# ------------------------------------------------------------------ work
def work(case):
    c = case
    p1, cells = c["degree"] + 1, c["nx"] * c["nz"]
    nq, nd = 2 * c["degree"] + 1, (c["degree"] + 1) ** 2
    n = cells * nd
    line = p1 * nq  # multiply-adds of one 1D contraction, halved by the basis's symmetry
    interp = (p1 + nq) * line  # flops of one field's values at the points
    points = nq * nq
    s = c["stage"]
    rhs_fields = 4 * s + 3

    def rhs_flops():  # values in, four outputs tested with phi and both derivatives, the fluxes, four faces
        return cells * (rhs_fields * interp + 4 * (2 * line * nq + 2 * line * p1) + 45 * s * points
                        + 4 * nq * (8 * s * p1 + 55 * s) / 2)

    apply_b = {"bytes": 8 * 3 * n, "flops": cells * (3 * interp + 8 * p1**3)}
    apply_c = {"bytes": 8 * 4 * n, "flops": cells * (5 * interp + 12 * points)}
    schur = {"bytes": 8 * 4 * n, "flops": apply_b["flops"] + apply_c["flops"] + 4 * cells * nd * nd}
    if c["kind"] in ("rhs", "rhs_split"):
        return {"bytes": 8 * n * (rhs_fields + 4), "flops": rhs_flops()}
    if c["kind"] == "backward":
        return {"bytes": 8 * n * (2 * rhs_fields + 4), "flops": 3 * rhs_flops()}
    if c["kind"] == "tangent":
        return {"bytes": 8 * n * (2 * rhs_fields + 4), "flops": 2 * rhs_flops()}
    if c["kind"] == "implicit":
        inverse = cells * nd**3 / 3
        return {"bytes": 8 * n * 22, "flops": apply_b["flops"] + apply_c["flops"] + schur["flops"] + inverse
                + 8 * cells * nd * nd}
    # iterations at this time step: 15 of degree 16 (polynomial), 30 cycles, 150 (Jacobi); a polynomial's step reads
    # and writes its direction, its residual and its iterate in 32 bits
    inner = {"bytes": 4 * 8 * n, "flops": cells * 40 * p1**3}
    its, steps = {"cheb_fp32": (15, 16), "cheb_fp64": (15, 16), "mg_fp32": (30, 14), "mg_fp64": (30, 14)}.get(
        c["precond"], (150, 0))
    if c["kind"] == "solve":
        return {k: its * (schur[k] + steps * inner[k]) for k in ("bytes", "flops")}
    per_step = {"cheb_fp32": (21, 20), "jacobi": (350, 0), "default": (40, 0)}[c["precond"]]
    w = {k: per_step[0] * (schur[k] + per_step[1] * inner[k]) + {"bytes": 8 * 120 * n, "flops": 3 * cells * 3e4}[k]
         for k in ("bytes", "flops")}
    return {k: 4 * v for k, v in w.items()} if c["kind"] == "imex_grad" else w


# ------------------------------------------------------------------ 64-bit evaluation in plain torch
class _Dense:
    """The discontinuous Galerkin operators by dense 1D matrices on (nz, nx, P+1, P+1) arrays."""

    def __init__(self, c):
        self.c = c
        self.dev = torch.device("cuda")
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        p, nq = c["degree"], 2 * c["degree"] + 1
        self.P, self.nq = p, nq
        s = _gll(p)
        g, w = np.polynomial.legendre.leggauss(nq)
        g, w = 0.5 * (g + 1.0), 0.5 * w
        S, D = np.ones((nq, p + 1)), np.zeros((nq, p + 1))
        for i in range(p + 1):
            others = [j for j in range(p + 1) if j != i]
            for j in others:
                S[:, i] *= (g - s[j]) / (s[i] - s[j])
            for j in others:
                term = np.full(nq, 1.0 / (s[i] - s[j]))
                for k in others:
                    if k != j:
                        term *= (g - s[k]) / (s[i] - s[k])
                D[:, i] += term
        self.S, self.D, self.w = t(S), t(D), t(w)
        V = t(_vertices(c))
        v0, v1, v2, v3 = V[:-1, :-1], V[:-1, 1:], V[1:, :-1], V[1:, 1:]
        xi, eta = t(g)[None, None, None, :], t(g)[None, None, :, None]
        e = lambda a: a[:, :, None, None]  # noqa: E731
        bil = v3 - v2 - v1 + v0
        self.J00, self.J10 = e((v1 - v0)[..., 0]) + eta * e(bil[..., 0]), e((v1 - v0)[..., 1]) + eta * e(bil[..., 1])
        self.J01, self.J11 = e((v2 - v0)[..., 0]) + xi * e(bil[..., 0]), e((v2 - v0)[..., 1]) + xi * e(bil[..., 1])
        self.ww = self.w[:, None] * self.w[None, :]
        self.dw = (self.J00 * self.J11 - self.J01 * self.J10) * self.ww
        self.X = [e(v0[..., k]) + xi * e((v1 - v0)[..., k]) + eta * e((v2 - v0)[..., k]) + xi * eta * e(bil[..., k]) for k in (0, 1)]
        tr, tt, tl, tb = v3 - v1, v3 - v2, v2 - v0, v1 - v0
        unit = lambda a, b: (a / torch.sqrt(a * a + b * b), b / torch.sqrt(a * a + b * b))  # noqa: E731
        length = lambda q: torch.sqrt(q[..., 0] ** 2 + q[..., 1] ** 2)[:, :, None] * self.w  # noqa: E731
        # outward normals of the right and top faces, and of the left and bottom ones for the walls
        f = lambda q: tuple(x[:, :, None] for x in q)  # noqa: E731
        self.n_r, self.n_t = f(unit(tr[..., 1], -tr[..., 0])), f(unit(-tt[..., 1], tt[..., 0]))
        self.n_l, self.n_b = f(unit(-tl[..., 1], tl[..., 0])), f(unit(tb[..., 1], -tb[..., 0]))
        self.l_r, self.l_t, self.l_l, self.l_b = length(tr), length(tt), length(tl), length(tb)
        self.periodic = c["mesh"] == "annulus" or c["periodic"]

    def split(self, v, comps):
        p1 = self.P + 1
        v = v.reshape(self.c["nz"], self.c["nx"], comps, p1, p1)
        return [v[:, :, k] for k in range(comps)]

    def join(self, fields):
        return torch.stack(fields, dim=2).reshape(-1)

    def at(self, f):
        return self.S @ f @ self.S.T

    def test(self, val=None, grad=None):
        """int val phi + grad . nabla phi"""
        out = 0.0
        if val is not None:
            out = self.S.T @ (val * self.dw) @ self.S
        if grad is not None:
            gx, gz = grad
            fx, fe = (self.J11 * gx - self.J01 * gz) * self.ww, (self.J00 * gz - self.J10 * gx) * self.ww
            out = out + self.S.T @ fx @ self.D + self.D.T @ fe @ self.S
        return out

    def faces(self, fields, flux, wall=None):
        """The face terms: flux(inside, outside, n) per output, tested with minus the inside's and plus the
        outside's basis; wall(inside, n) per output, tested with plus the inside's."""
        P, S = self.P, self.S
        nz, nx = self.c["nz"], self.c["nx"]
        side = {"l": lambda f: f[..., :, 0] @ S.T, "r": lambda f: f[..., :, P] @ S.T, "b": lambda f: f[..., 0, :] @ S.T,
                "t": lambda f: f[..., P, :] @ S.T}
        out = None

        def add(parts, which):
            nonlocal out
            out = [torch.zeros(nz, nx, P + 1, P + 1, dtype=torch.float64, device=self.dev) for _ in parts] if out is None else out
            for o, g in zip(out, parts):
                t = g @ S
                if which == "l":
                    o[..., :, 0] += t
                elif which == "r":
                    o[..., :, P] += t
                elif which == "b":
                    o[..., 0, :] += t
                else:
                    o[..., P, :] += t

        keep = torch.ones(nz, nx, 1, dtype=torch.float64, device=self.dev)
        keep_x, keep_z = keep.clone(), keep.clone()
        if not self.periodic:
            keep_x[:, -1] = 0.0
        keep_z[-1] = 0.0
        for a, b, n, ln, k, dim in (("r", "l", self.n_r, self.l_r, keep_x, 1), ("t", "b", self.n_t, self.l_t, keep_z, 0)):
            ins = [side[a](f) for f in fields]
            outs = [torch.roll(side[b](f), -1, dim) for f in fields]
            F = [g * ln * k for g in flux(ins, outs, n)]
            add([-g for g in F], a)
            add([torch.roll(g, 1, dim) for g in F], b)
        if wall is not None:
            for a, n, ln, k in (("r", self.n_r, self.l_r, 1.0 - keep_x), ("t", self.n_t, self.l_t, 1.0 - keep_z),
                                ("l", self.n_l, self.l_l, torch.roll(1.0 - keep_x, 1, 1)),
                                ("b", self.n_b, self.l_b, torch.roll(1.0 - keep_z, 1, 0))):
                add([g * ln * k for g in wall([side[a](f) for f in fields], n)], a)
        return out

    # --- explicit right-hand sides
    def rhs(self, src):
        c, dt = self.c, _dt(self.c)
        s, Ma2 = c["stage"], MA * MA
        iM, iF = 1.0 / Ma2, 1.0 / (FR * FR)
        g = 2.0 - math.sqrt(2.0)
        q = math.sqrt(2.0) / 4.0
        ca = {1: [g], 2: [0.5, 0.5], 3: [q, q, 1.0 - 2.0 * q]}[s]
        ct = {1: [g / 2], 2: [q, q], 3: ca}[s]
        cg, cI = ct, {1: g / 2, 2: 1.0 - 2.0 * q, 3: 0.0}[s]
        ca, ct, cg, cI = [a * dt for a in ca], [a * dt for a in ct], [a * dt for a in cg], cI * dt
        if c["mesh"] == "annulus":
            r2 = self.X[0] ** 2 + self.X[1] ** 2
            e0, e1 = (self.X[k] / torch.sqrt(r2) * (EARTH**2 / r2) for k in (0, 1))
        else:
            e0, e1 = 0.0, 1.0
        tau = None
        if c.get("sponge"):
            z0, z1, rate, x0, x1, width, lat, u_ref = SPONGE
            up = rate * torch.sin(0.5 * math.pi * (self.X[1] - z0) / (z1 - z0)) ** 2
            d = torch.minimum(self.X[0] - x0, x1 - self.X[0])
            tau = torch.where(self.X[1] > z0, up, 0.0) + torch.where(d < width, lat * torch.cos(0.5 * math.pi * d / width) ** 2, 0.0)
        total = [0.0, 0.0, 0.0, 0.0]
        u0 = self.split(src[1], 2)
        for j in range(s):
            rho, p = self.split(src[3 * j], 1)[0], self.split(src[3 * j + 2], 1)[0]
            ux, uz = self.split(src[3 * j + 1], 2)
            R, U, W, Q = self.at(rho), self.at(ux), self.at(uz), self.at(p)
            uu = U * U + W * W
            vx, vz = -cg[j] * iF * R * e0, -cg[j] * iF * R * e1
            if tau is not None:
                vx = vx - ca[j] * tau * R * (U - SPONGE[7])
                vz = vz - ca[j] * tau * R * W
            ve = -cg[j] * Ma2 * iF * R * (U * e0 + W * e1)
            vr = None
            if j == 0:
                vr, vx, vz, ve = R, vx + R * U, vz + R * W, ve + G1 * Q + 0.5 * Ma2 * R * uu
            pt = ct[j] * iM * Q
            k = 0.5 * ca[j] * Ma2 * uu * R + ct[j] * GG * Q
            cells = [self.test(vr, (ca[j] * R * U, ca[j] * R * W)),
                     self.test(vx, (ca[j] * R * U * U + pt, ca[j] * R * U * W)),
                     self.test(vz, (ca[j] * R * W * U, ca[j] * R * W * W + pt)), self.test(ve, (k * U, k * W))]
            quirk = s == 2 and j == 1  # the reference's kinetic jump u_tmp_2 . u_old

            def flux(a, b, n, j=j, quirk=quirk):
                an, bn = a[1] * n[0] + a[2] * n[1], b[1] * n[0] + b[2] * n[1]
                lam = torch.maximum(an.abs(), bn.abs())
                half = 0.5 * ca[j]
                pa = 0.5 * ct[j] * iM * (a[3] + b[3])
                ka, kb = a[1] ** 2 + a[2] ** 2, b[1] ** 2 + b[2] ** 2
                kin = 0.25 * (ka * a[0] * an + kb * b[0] * bn)
                ent = 0.5 * GG * (a[3] * an + b[3] * bn)
                if s < 3:
                    if quirk:
                        jk = 0.5 * (a[0] * (a[1] * a[4] + a[2] * a[5]) - b[0] * (b[1] * b[4] + b[2] * b[5]))
                    else:
                        jk = 0.5 * (a[0] * ka - b[0] * kb)
                    fe = ca[j] * Ma2 * (kin + 0.5 * lam * jk) + ct[j] * (ent + 0.5 * lam * G1 * (a[3] - b[3]))
                else:
                    fe = ca[j] * (Ma2 * kin + ent + 0.5 * lam * (G1 * (a[3] - b[3]) + 0.5 * Ma2 * (a[0] * ka - b[0] * kb)))
                return [half * (a[0] * an + b[0] * bn + lam * (a[0] - b[0])),
                        half * (a[0] * a[1] * an + b[0] * b[1] * bn + lam * (a[0] * a[1] - b[0] * b[1])) + pa * n[0],
                        half * (a[0] * a[2] * an + b[0] * b[2] * bn + lam * (a[0] * a[2] - b[0] * b[2])) + pa * n[1], fe]

            def wall(a, n, j=j):
                z = ct[j] * iM * a[3]
                return [0.0 * z, -z * n[0], -z * n[1], 0.0 * z]

            fields = [rho, ux, uz, p] + (u0 if quirk else [])
            total = [x + y + z for x, y, z in zip(total, cells, self.faces(fields, flux, wall))]
        R = self.at(self.split(src[3 * s], 1)[0])
        U, W = (self.at(x) for x in self.split(src[3 * s + 1], 2))
        ve = -0.5 * Ma2 * R * (U * U + W * W)
        if s < 3:
            ve = ve - cI * Ma2 * iF * R * (U * e0 + W * e1)
            total[1] = total[1] + self.test(-cI * iF * R * e0)
            total[2] = total[2] + self.test(-cI * iF * R * e1)
        total[3] = total[3] + self.test(ve)
        return [total[0].reshape(-1), self.join(total[1:3]), total[3].reshape(-1)]

    # --- implicit operators
    def coeff(self):
        return (1.0 - math.sqrt(2.0) / 2.0) if self.c["stage"] != 1 else 0.5 * (2.0 - math.sqrt(2.0))

    def B(self, p):
        k = self.coeff() * _dt(self.c) / (MA * MA)
        f = self.split(p, 1)[0]
        v = -k * self.at(f)
        zero = torch.zeros_like(v)
        cell = [self.test(None, (v, zero)), self.test(None, (zero, v))]
        flux = lambda a, b, n: [-0.5 * k * (a[0] + b[0]) * n[0], -0.5 * k * (a[0] + b[0]) * n[1]]  # noqa: E731
        wall = lambda a, n: [k * a[0] * n[0], k * a[0] * n[1]]  # noqa: E731
        return self.join([x + y for x, y in zip(cell, self.faces([f], flux, wall))])

    def C(self, w, pf):
        k = self.coeff() * _dt(self.c)
        wx, wz = self.split(w, 2)
        f = self.split(pf, 1)[0]
        v = -k * GG * self.at(f)
        cell = self.test(None, (v * self.at(wx), v * self.at(wz)))

        def flux(a, b, n):
            an, bn = a[0] * n[0] + a[1] * n[1], b[0] * n[0] + b[1] * n[1]
            lam = torch.maximum(an.abs(), bn.abs())
            return [-k * (0.5 * GG * (a[2] * an + b[2] * bn) + 0.5 * lam * G1 * (a[2] - b[2]))]

        return (cell + self.faces([wx, wz, f], flux)[0]).reshape(-1)

    def mass(self, weight=None):
        """Cell mass matrices (cells, ND, ND), weighted."""
        f = self.dw if weight is None else self.dw * self.at(self.split(weight, 1)[0])
        nd = (self.P + 1) ** 2
        phi = torch.einsum("qi,rj->qrij", self.S, self.S).reshape(self.nq**2, nd)
        out = torch.empty(self.c["nz"] * self.c["nx"], nd, nd, dtype=torch.float64, device=self.dev)
        f = f.reshape(-1, self.nq**2)
        for k in range(0, f.shape[0], 4096):
            out[k:k + 4096] = torch.einsum("qi,cq,qj->cij", phi, f[k:k + 4096], phi) if nd <= 9 else (phi.T * f[k:k + 4096, None, :]) @ phi
        return out

    def cells(self, mats, v, comps):
        return (v.reshape(mats.shape[0], comps, -1) @ mats.transpose(1, 2)).reshape(-1)

    def schur(self, Ainv, pf, p):
        D = G1 * self.test(self.at(self.split(p, 1)[0])).reshape(-1)
        return D - self.C(self.cells(Ainv, self.B(p), 2), pf)


def _solve(m, d):
    """The Schur system by BiCGStab on D^{-1} S with residual corrections (S is linear up to its wave-speed term)."""
    Ainv = torch.linalg.inv(m.mass(d["rho"]))
    Dinv = torch.linalg.inv(m.mass()) / G1
    S = lambda p: m.schur(Ainv, d["pf"], p)  # noqa: E731
    pre = lambda r: m.cells(Dinv, r, 1)  # noqa: E731
    x = torch.zeros_like(d["b"])
    for _ in range(12):
        r0 = d["b"] - S(x)
        if float(r0.norm()) < 3e-13 * float(d["b"].norm()):
            break
        e, r = torch.zeros_like(x), pre(r0)
        goal, hat = 1e-5 * float(r.norm()), r.clone()
        rho = alpha = omega = 1.0
        v = q = torch.zeros_like(x)
        for _ in range(600):
            rho, old = float(hat @ r), rho
            q = r + (rho / old) * (alpha / omega) * (q - omega * v)
            v = pre(S(q))
            alpha = rho / float(hat @ v)
            s = r - alpha * v
            t = pre(S(s))
            omega = float(t @ s) / float(t @ t)
            e += alpha * q + omega * s
            r = s - omega * t
            if not float(r.norm()) > goal:
                break
        x += e
    return x


def exact(case, seed):
    """What `run` returns, in 64 bits by plain torch; None for whole time steps (their nested solves take minutes)."""
    c = case
    nodes = c["nx"] * c["nz"] * (c["degree"] + 1) ** 2
    if c["kind"] in ("imex", "imex_grad") or (c["kind"] == "solve" and nodes > 9e5):
        return None
    d, m = _inputs(c, seed), _Dense(c)
    if c["kind"] in ("rhs", "rhs_split"):
        return m.rhs(d["src"])
    if c["kind"] == "backward":
        src = [x.requires_grad_() for x in d["src"]]
        return list(torch.autograd.grad(m.rhs(src), src, d["ybar"]))
    if c["kind"] == "tangent":
        src = [x.requires_grad_() for x in d["src"]]
        y = m.rhs(src)
        dummy = [torch.zeros_like(t, requires_grad=True) for t in y]
        back = torch.autograd.grad(y, src, dummy, create_graph=True)
        return list(torch.autograd.grad(back, dummy, d["dsrc"]))
    if c["kind"] == "solve":
        return _solve(m, d)
    A, M = m.mass(d["rho"]), m.mass()
    Ainv = torch.linalg.inv(A)
    return {"B": m.B(d["p"]), "C": m.C(d["w"], d["pf"]), "A": m.cells(A, d["v"], 2), "Ainv": m.cells(Ainv, d["v"], 2),
            "Minv": m.cells(torch.linalg.inv(M), d["r"], 1), "schur": m.schur(Ainv, d["pf"], d["p"])}
