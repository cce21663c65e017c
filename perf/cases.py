"""The work a user of this package has it do, as measured cases.

A case is a dict of plain values; ``kind`` says which public entry point a pass goes through:

  step      Sod2dMesh.rk_4_main, one RK4 step (the call of a SOD2D time loop)
  steps     Sod2dMesh.rk4_steps, ``steps`` graph-replayed steps in one call
  rhs       Sod2dMesh.rhs, the stage right-hand side
  vjp       Sod2dMesh.rhs_vjp, its adjoint
  rollout   Sod2dRollout.apply + backward: ``steps`` steps and the gradient of 1/2 |rho u|^2
  routines  full_convec_ijk, full_diffusion_ijk and generic_scalar_convec_ijk (the per-routine drop-ins)
  pcg       Sod2dPoisson.solve, the pressure Poisson CG to a relative residual of 1e-10
  ensemble  Sod2dBatch.rk4_steps on ``members`` uneven boxes, then every member read back

Meshes are n^3 HEX64 boxes with jittered nodes: triply periodic with a perturbed Taylor-Green
vortex, or (flow = "channel") walls in y with a driven shear profile.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from sod2d_refmap_b200 import mesh as M
from sod2d_refmap_b200.adjoint import Sod2dRollout
from sod2d_refmap_b200.solver import FP64, MIXED, Sod2dBatch, Sod2dMesh, Sod2dPoisson, Sod2dState

DRIVE = 0.05  # momentum source of the channel


def _case(kind, n, precision="fp64", option="none", flow="tgv", steps=1, members=0, name=None):
    c = dict(kind=kind, n=n, precision=precision, option=option, flow=flow, steps=steps, members=members)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the package's headline run: one mixed-precision time step of the 64^3 vortex (7.1 M nodes)
        _case("step", 64, "mixed", name="step_mixed_64"),
        # the same loop in full precision at the size of the adjoint configuration
        _case("step", 32, "fp64", name="step_fp64_32"),
        # the 8^3 configuration: a coarse run or a regression test, where launches and latency count
        _case("step", 8, "mixed", name="step_mixed_8"),
        # a large-eddy run advanced many steps per call
        _case("steps", 24, "mixed", option="les", steps=10, name="steps_mixed_les_24"),
        # a wall-bounded flow: no-slip walls and a constant driving force, odd element count
        _case("step", 15, "fp64", flow="channel", name="step_fp64_channel_15"),
        # the right-hand side alone, as an outer integrator of the user's own calls it
        _case("rhs", 21, "mixed", name="rhs_mixed_21"),
        _case("rhs", 33, "fp64", option="enthalpy", name="rhs_fp64_enthalpy_33"),
        # sensitivities: one reverse product, and a whole differentiated rollout
        _case("vjp", 27, "fp64", name="vjp_fp64_27"),
        _case("rollout", 32, "mixed", steps=10, name="rollout_mixed_32"),
        # SOD2D's own routines replaced one by one
        _case("routines", 20, "fp64", name="routines_fp64_20"),
        # the incompressible pressure solve
        _case("pcg", 24, "fp64", name="pcg_fp64_24"),
        # a parameter study: many small uneven boxes at once
        _case("ensemble", 24, "mixed", steps=40, members=8, name="ensemble_mixed_24"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "steps", "rhs", "rhs", "vjp", "rollout", "routines", "pcg", "ensemble"])
    precision = rng.choice(["fp64", "mixed"])
    option = rng.choice(["none", "none", "les", "enthalpy"])
    if kind == "step":
        flow = rng.choice(["tgv", "tgv", "channel"])
        return _case(kind, _log_int(rng, 4, 48), precision, option, flow)
    if kind == "steps":
        return _case(kind, _log_int(rng, 4, 24), precision, option, "tgv", rng.randint(2, 20))
    if kind == "rhs":
        return _case(kind, _log_int(rng, 4, 48), precision, "enthalpy" if option == "enthalpy" else "none")
    if kind == "vjp":
        return _case(kind, _log_int(rng, 4, 36), "fp64", "enthalpy" if option == "enthalpy" else "none")
    if kind == "rollout":
        return _case(kind, _log_int(rng, 4, 24), precision, option, "tgv", rng.randint(2, 12))
    if kind == "routines":
        return _case(kind, _log_int(rng, 4, 40), "fp64")
    if kind == "pcg":
        return _case(kind, _log_int(rng, 4, 32), precision)
    return _case(kind, rng.randint(6, 24), precision, "none", "tgv", rng.randint(10, 40), rng.randint(2, 8))


# ---- inputs --------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _box(n, flow):
    """The mesh arrays a SOD2D run reads from its mesh file."""
    if flow == "channel":
        return M.channel_box(n, jitter=0.05, seed=11, codes=(M.BC_NON_SLIP_ADIABATIC, M.BC_NON_SLIP_ADIABATIC))
    return M.periodic_box(n, jitter=0.05, seed=11)


def _params(case):
    return M.TGVParams(flag_les=int(case["option"] == "les"), flag_total_enthalpy=int(case["option"] == "enthalpy"))


def _precision(case):
    return MIXED if case["precision"] == "mixed" else FP64


def _primitive(box, prm, flow, seed):
    """rho, u (3, npoin), p and mu_factor of the initial state on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    x, y, z = (torch.from_numpy(np.ascontiguousarray(box.coord[:, c])).cuda() for c in range(3))
    noise = 2.0 * torch.rand(3, x.numel(), dtype=torch.float64, device="cuda", generator=g) - 1.0
    if flow == "channel":
        s = 2.0 * y / box.L - 1.0
        u = torch.stack([1.5 * (1.0 - s * s) + 0.1 * (1.0 - s * s) * torch.sin(2 * z), 0.1 * (1.0 - s * s) * torch.sin(x),
                         0.1 * (1.0 - s * s) * torch.cos(x)])
        u = u + 1e-3 * (1.0 - s * s) * noise
        p = torch.full_like(x, prm.p0)
    else:
        u = torch.stack([torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z),
                         torch.zeros_like(x)]) + 1e-3 * noise
        p = prm.p0 + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
    rho = p / (prm.Rgas * prm.T0)
    return rho, u, p, torch.full_like(x, prm.mu_factor), g


def _state(case, seed):
    """The arrays of a running simulation: conserved and primitive fields, the viscosities the step
    before left, and its time step."""
    box, prm = _box(case["n"], case["flow"]), _params(case)
    rho, u, p, mf, g = _primitive(box, prm, case["flow"], seed)
    s = Sod2dState(box.npoin, box.nelem)
    gam = prm.gamma_gas
    s.rho.copy_(rho); s.u.copy_(u); s.q.copy_(rho * u); s.pr.copy_(p)
    s.E.copy_(p / (gam - 1.0) + 0.5 * rho * (u * u).sum(0))
    s.Tem.copy_(p / (rho * prm.Rgas)); s.e_int.copy_(p / (rho * (gam - 1.0)))
    s.csound.copy_(torch.sqrt(gam * p / rho)); s.eta.copy_(rho / (gam - 1.0) * torch.log(p / rho ** gam))
    s.machno.copy_((u * u).sum(0) / s.csound); s.mu_factor.copy_(mf)
    s.mu_fluid.copy_(_sutherland(s.Tem, mf))
    s.mu_e.copy_(1e-4 * torch.rand(64, box.nelem, dtype=torch.float64, device="cuda", generator=g))
    if prm.flag_les:
        s.mu_sgs.copy_(1e-5 * torch.rand(64, box.nelem, dtype=torch.float64, device="cuda", generator=g))
    s.dt.fill_(0.5 * (box.L / box.n) / 7.0 / 12.0)
    return box, prm, s


def _channel(handle, box):
    handle.set_boundaries(box.extra["bou_codes_nodes"], box.extra["lnbn_nodes"], box.extra["normals"])
    src = torch.zeros(3, box.npoin, dtype=torch.float64, device="cuda")
    src[0] = DRIVE
    handle.set_source_term(src)


def _seeds(box, seed):
    """Seed vectors of the reverse product and the Poisson right-hand side."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
    return torch.randn(5, box.npoin, dtype=torch.float64, device="cuda", generator=g)


def _members(case, seed):
    """The ensemble: sides 4..n log-uniformly, each with its own state and Reynolds number."""
    rng = random.Random(1000 * case["members"] + case["n"])
    prm = _params(case)
    boxes = [_member_box(_log_int(rng, 4, case["n"])) for _ in range(case["members"])]
    res = [400.0 * 8.0 ** rng.random() for _ in boxes]
    states = [M.taylor_green_state(b, prm, 1e-3, seed=int(seed) * 64 + i, re=r) for i, (b, r) in enumerate(zip(boxes, res))]
    dts = [0.5 * (b.L / b.n) / 7.0 / 12.0 for b in boxes]
    return prm, boxes, states, dts


@functools.lru_cache(maxsize=16)
def _member_box(n):
    return M.periodic_box(n, jitter=0.05, seed=11)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        prm, boxes, states, dts = _members(case, seed)
        batch = Sod2dBatch(boxes, states, prm)
        batch.set_dt(dts)
        return dict(case=case, batch=batch)
    box, prm, s = _state(case, seed)
    handle = Sod2dMesh(box, prm)
    if case["flow"] == "channel":
        _channel(handle, box)
    st = dict(case=case, mesh=handle, state=s)
    if kind == "vjp":
        st["bar"] = _seeds(box, seed)
    if kind == "pcg":
        st["poisson"] = Sod2dPoisson(handle)
        b = _seeds(box, seed)[0]
        st["rhs"] = b - b.mean()
    if kind == "rollout":
        s.mu_e.zero_(); s.mu_sgs.zero_()
    return st


# ---- one pass ------------------------------------------------------------------------------------
STATE = ("rho", "q", "E", "u", "pr", "Tem", "e_int", "eta", "csound", "machno", "mu_fluid", "mu_e", "Reta")


def _outputs(s, les):
    out = {f: getattr(s, f) for f in STATE + (("mu_sgs",) if les else ())}
    out["dt"] = s.dt
    return out


def run(st):
    case = st["case"]
    kind, prec = case["kind"], _precision(case)
    if kind == "ensemble":
        st["batch"].rk4_steps(case["steps"], prec)
        got = [st["batch"].get_member(i) for i in range(case["members"])]
        out = {f: np.concatenate([g[f] for g in got]) for f in STATE}
        out["dt"] = st["batch"].dt()
        return out
    mesh, s = st["mesh"], st["state"]
    if kind == "step":
        mesh.rk_4_main(s, prec)
        return _outputs(s, case["option"] == "les")
    if kind == "steps":
        mesh.rk4_steps(s, case["steps"], prec)
        return _outputs(s, case["option"] == "les")
    if kind == "rhs":
        return mesh.rhs(s, prec)
    if kind == "vjp":
        b = st["bar"]
        return mesh.rhs_vjp(s.rho, s.q, s.E, s.mu_e, s.mu_factor, b[0], b[1:4], b[4])
    if kind == "routines":
        conv = mesh.full_convec_ijk(s.u, s.q, s.rho, s.pr, s.e_int)
        diff = mesh.full_diffusion_ijk(s.rho, s.rho, s.u, s.Tem, s.mu_fluid, s.mu_e)
        return conv, diff, mesh.generic_scalar_convec_ijk(s.q, s.eta, s.u)
    if kind == "pcg":
        return st["poisson"].solve(st["rhs"], tol=1e-10, mixed=case["precision"] == "mixed")[0]
    x = [t.clone().requires_grad_(True) for t in (s.rho, s.q, s.E)]
    y = Sod2dRollout.apply(mesh, s, *x, case["steps"], 10, precision=prec)
    (0.5 * (y[1] * y[1]).sum()).backward()
    return [t.detach() for t in y], [t.grad for t in x]


# ---- what a pass cannot do without -----------------------------------------------------------------
RHS_FLOPS = 900.0    # per gauss point and stage: split convection, gradients, viscous fluxes, divergence
VJP_FLOPS = 2200.0   # per gauss point: the forward quantities and the reverse sweep


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        rng = random.Random(1000 * case["members"] + case["n"])
        sides = [_log_int(rng, 4, case["n"]) for _ in range(case["members"])]
        E, N = sum(n ** 3 for n in sides), sum((3 * n) ** 3 for n in sides)
    else:
        n = case["n"]
        E, N = n ** 3, (3 * n) ** 2 * (3 * n + (case["flow"] == "channel"))
    P = 64 * E
    real = 4 if case["precision"] == "mixed" else 8
    fixed = P * (10 * real + 4)  # the metric terms and the connectivity
    if kind in ("step", "steps", "ensemble"):
        les = 2 if case["option"] == "les" else 0
        return dict(bytes=fixed + 8 * (22 * N + (2 + les) * P), flops=case["steps"] * 4 * RHS_FLOPS * P)
    if kind == "rhs":
        return dict(bytes=fixed + 8 * (12 * N + P), flops=RHS_FLOPS * P)
    if kind == "vjp":
        return dict(bytes=fixed + 8 * (16 * N + P), flops=VJP_FLOPS * P)
    if kind == "routines":
        return dict(bytes=fixed + 8 * (24 * N + P), flops=RHS_FLOPS * P)
    if kind == "pcg":  # about 23 n iterations on these meshes, each one product on a 6-value metric
        it = 23 * n
        return dict(bytes=it * (P * (6 * real + 4) + 9 * real * N), flops=it * (70.0 * P + 12.0 * N))
    return dict(bytes=fixed + 8 * (16 * N + P), flops=case["steps"] * 4 * (RHS_FLOPS + VJP_FLOPS) * P)


def tolerance(case):
    """About four times the distance from the 64-bit values over all outputs of a case: the mixed
    path's FP32 element arithmetic shows up to 2.7e-6 (the entropy residual), FP64 2.6e-12 (the
    momentum residual, whose pressure gradient cancels), a CG stopped at 1e-10 up to 3e-10; a rollout's
    gradients average the FP32 rounding (8e-8)."""
    if case["kind"] == "pcg":
        return {"rel": 2e-9}
    if case["precision"] == "fp64":
        return {"rel": 2e-11}
    return {"rel": 1e-6 if case["kind"] == "rollout" else 1e-5}


# ---- the same in 64 bits, in plain torch -----------------------------------------------------------
def _sutherland(T, mf):
    return mf * 0.000001458 * T ** 1.5 / (T + 110.4)


class _Ref:
    """Geometry and operators of one mesh on (nelem, k, j, i) arrays, in the reference's formulas."""

    def __init__(self, box, prm):
        self.box, self.prm = box, prm
        T = box.tables
        d_of_a = T.nat_ijk[:, 0] + 4 * T.nat_ijk[:, 1] + 16 * T.nat_ijk[:, 2]
        self.a_of_d = torch.from_numpy(np.argsort(d_of_a)).cuda()
        order = np.argsort(d_of_a)
        self.conn = torch.from_numpy(np.ascontiguousarray(box.connec[:, order]).astype(np.int64)).cuda()
        orig = torch.from_numpy(np.ascontiguousarray(box.connec_orig[:, order]).astype(np.int64)).cuda()
        self.E, self.N = box.nelem, box.npoin
        self.D = torch.from_numpy(T.D.copy()).cuda()
        xyz = [torch.from_numpy(np.ascontiguousarray(box.coord_orig[:, c])).cuda()[orig].view(-1, 4, 4, 4) for c in range(3)]
        J = torch.stack([torch.stack(self.iso(x)) for x in xyz])  # J[c][r] = dx_c / dxi_r
        Jm = J.permute(2, 3, 4, 5, 0, 1)
        self.H = torch.linalg.inv(Jm).transpose(-1, -2).permute(4, 5, 0, 1, 2, 3).contiguous()  # H[c][r] = dxi_r / dx_c
        det = torch.linalg.det(Jm)
        w = torch.from_numpy(M.gll_nodes_weights()[1]).cuda()
        self.gpv = w[:, None, None] * w[None, :, None] * w[None, None, :] * det
        self.Ml = self.scatter(self.gpv)
        pts = torch.stack(xyz, -1).view(self.E, 64, 3)
        self.hl = torch.empty(self.E, 64, dtype=torch.float64, device="cuda")
        eye = 1e12 * torch.eye(64, dtype=torch.float64, device="cuda")
        for b in range(0, self.E, 8192):
            q = pts[b:b + 8192]
            r2 = sum((q[:, :, None, c] - q[:, None, :, c]) ** 2 for c in range(3))
            self.hl[b:b + 8192] = (r2 + eye).amin(-1).sqrt()
        self.hl = self.hl.view(-1, 4, 4, 4)
        cor = torch.stack(xyz, -1)[:, ::3, ::3, ::3]  # corners (E, 2, 2, 2, 3)
        self.he = torch.stack([(cor.select(a, 1) - cor.select(a, 0)).norm(dim=-1).reshape(self.E, 4).amin(1)
                               for a in (1, 2, 3)]).amin(0)
        dmin, dmax = det.reshape(self.E, 64).amin(1), det.reshape(self.E, 64).amax(1)
        self.jratio = (dmin / dmax) ** 2
        self.wall = None
        if "bou_codes_nodes" in box.extra:
            self.wall = torch.from_numpy(box.extra["bou_codes_nodes"] < M.MAX_NUM_BOU_CODES).cuda()

    def iso(self, f):
        D = self.D
        return (torch.einsum("im,ekjm->ekji", D, f), torch.einsum("jm,ekmi->ekji", D, f), torch.einsum("km,emji->ekji", D, f))

    def grad(self, f):
        g = self.iso(f)
        return [sum(self.H[c][r] * g[r] for r in range(3)) for c in range(3)]

    def div(self, v):
        return sum(self.grad(v[c])[c] for c in range(3))

    def weak_div(self, v):
        """sum_q D[q][a] gpvol He^T v along the three lines through a."""
        F = [self.gpv * sum(self.H[c][r] * v[c] for c in range(3)) for r in range(3)]
        D = self.D
        return (torch.einsum("mi,ekjm->ekji", D, F[0]) + torch.einsum("mj,ekmi->ekji", D, F[1]) +
                torch.einsum("mk,emji->ekji", D, F[2]))

    def at(self, f):
        return f[self.conn].view(-1, 4, 4, 4)

    def scatter(self, r):
        return torch.zeros(self.N, dtype=torch.float64, device="cuda").index_add(0, self.conn.reshape(-1), r.reshape(-1))

    def internal(self, m):
        return m[self.a_of_d].t().reshape(-1, 4, 4, 4)

    def external(self, m):
        out = torch.empty(64, self.E, dtype=torch.float64, device="cuda")
        out[self.a_of_d] = m.reshape(self.E, 64).t()
        return out

    def convec(self, u, q, rho, p, E, total=None):
        """full_convec_ijk for an energy-like E (per mass); total: E + p of full_convec_ijk_H."""
        gr, dU, dQ = self.grad(rho), self.div(u), self.div(q)
        gu, gq, gp = [self.grad(c) for c in u], [self.grad(c) for c in q], self.grad(p)
        dot = lambda a, b: sum(x * y for x, y in zip(a, b))
        Rm = 0.5 * (dQ + rho * dU + dot(u, gr))
        Rmo = []
        for c in range(3):
            Rmo.append(0.25 * (self.div([q[c] * u[j] for j in range(3)]) + u[c] * dQ + q[c] * dU +
                               rho * self.div([u[c] * u[j] for j in range(3)]) + u[c] * dot(u, gr) + dot(q, gu[c]) +
                               dot(u, gq[c])) + gp[c])
        if total is not None:
            Re = 0.5 * (self.div([total * c for c in u]) + total * dU + dot(u, self.grad(total)))
        else:
            Re = 0.0
            for e in (E, 0.5 * dot(u, u)):
                Re = Re + 0.25 * (self.div([rho * e * c for c in u]) + e * dQ + rho * e * dU + rho * self.div([e * c for c in u]) +
                                  dot(q, self.grad(e)) + dot(u, self.grad(rho * e)) + e * dot(u, gr))
        return [self.gpv * r for r in (Rm, *Rmo, Re)]

    def scalar(self, eta, u, f):
        return self.gpv * 0.5 * (self.div(f) + eta * self.div(u) + sum(a * b for a, b in zip(u, self.grad(eta))))

    def diffusion(self, rho, u, T, muf, mue, mus):
        prm = self.prm
        gu, gr, gT = [self.grad(c) for c in u], self.grad(rho), self.grad(T)
        dU = gu[0][0] + gu[1][1] + gu[2][2]
        mf = muf + rho * mus
        tau = [[(mf + mue) * (gu[r][c] + gu[c][r]) - (mf * (2.0 / 3.0) * dU if r == c else 0.0) for c in range(3)] for r in range(3)]
        tu = [sum(tau[r][c] * u[c] for c in range(3)) for r in range(3)]
        nu = prm.c_rho * mue / rho
        kap = (muf + prm.c_ener * mue) * (prm.Cp / prm.Prt) + prm.Cp * rho * mus / 0.9
        return [nu * self.weak_div(gr), *(self.weak_div(t) for t in tau), self.weak_div(tu) + kap * self.weak_div(gT)]

    def rhs(self, rho, q, E, mf, mue, mus=None, eta=True):
        """The stage residuals (mass, momentum, energy, entropy) over the lumped mass."""
        prm = self.prm
        g = prm.gamma_gas
        r, qe, Ee = self.at(rho), [self.at(c) for c in q], self.at(E)
        u = [c / r for c in qe]
        k = 0.5 * sum(c * c for c in u)
        p = r * (g - 1.0) * (Ee / r - k)
        T = p / (r * prm.Rgas)
        tot = Ee + p if prm.flag_total_enthalpy else None
        mue = self.internal(mue)
        mus = self.internal(mus) if mus is not None else torch.zeros_like(mue)
        con = self.convec(u, qe, r, p, g / (g - 1.0) * p / r, tot)
        dif = self.diffusion(r, u, T, _sutherland(T, self.at(mf)), mue, mus)
        out = [self.scatter(a + b) / self.Ml for a, b in zip(con, dif)]
        if self.wall is not None:
            out[1] = out[1] - DRIVE
        if eta:
            ent = r / (g - 1.0) * torch.log(p / r ** g)
            out.append(self.scatter(self.scalar(ent, u, [ent * c for c in u])) / self.Ml)
        return out

    def walls(self, y):
        if self.wall is None:
            return y
        keep = (~self.wall).double()
        return [y[0] * keep + self.prm.rho0 * (1 - keep), *(y[c] * keep for c in (1, 2, 3)), y[4]]

    def advance(self, y, dt, mf, mue, mus=None):
        """The conserved fields after one RK4 step, and the entropy residual."""
        a, b = (0.0, 0.5, 0.5, 1.0), (1 / 6, 1 / 3, 1 / 3, 1 / 6)
        acc, r = [0.0] * 6, None
        for st in range(4):
            ys = self.walls(y if st == 0 else [y[f] - dt * a[st] * r[f] for f in range(5)])
            r = self.rhs(ys[0], ys[1:4], ys[4], mf, mue, mus)
            acc = [acc[f] + b[st] * r[f] for f in range(6)]
        new = self.walls([y[f] - dt * acc[f] for f in range(5)])
        reta = -acc[5]
        return new, (reta if self.wall is None else torch.where(self.wall, torch.zeros_like(reta), reta))

    def smooth(self, m):
        """The 3x3x3 (1/4, 1/2, 1/4) filter; the point past either end of a line is its second one."""
        W = torch.zeros(4, 4, dtype=torch.float64, device="cuda")
        for i in range(4):
            for j, w in ((i - 1, 0.25), (i, 0.5), (i + 1, 0.25)):
                W[i, j if 0 <= j <= 3 else 1] += w
        return torch.einsum("ia,jb,kc,ecba->ekji", W, W, W, m)

    def closure(self, y, reta, mf, mus):
        """Primitive fields, entropy viscosity, SGS viscosity and the next time step."""
        prm = self.prm
        g = prm.gamma_gas
        rho, E = y[0], y[4]
        u = torch.stack([c / rho for c in y[1:4]])
        um2 = (u * u).sum(0)
        ei = E / rho - 0.5 * um2
        p = rho * (g - 1.0) * ei
        cs, T = torch.sqrt(g * p / rho), p / (rho * prm.Rgas)
        eta = rho / (g - 1.0) * torch.log(p / rho ** g)
        mean = eta.mean()
        norm = torch.maximum(eta.max() - mean, mean - eta.min())
        out = dict(rho=rho, q=torch.stack(y[1:4]), E=E, u=u, pr=p, Tem=T, e_int=ei, eta=eta, csound=cs,
                   machno=um2.sqrt() / cs, mu_fluid=_sutherland(T, mf), Reta=reta)
        top = lambda f: f.reshape(self.E, 64).amax(1)
        vm, re, ue = self.at(um2.sqrt()), self.at(rho), [self.at(c) for c in u]
        he = self.he.view(-1, 1, 1, 1)
        M15 = (top(vm) / top(self.at(cs))) ** 15
        ced = torch.maximum((1.0 - self.jratio).clamp(min=prm.ce), torch.tanh(M15 * math.pi).clamp(min=prm.ce))
        beta = top(re * he * (prm.cmax / 3.0) * (vm + torch.sqrt(prm.Rgas * g * self.at(T))))
        R1 = re * self.at(reta).abs() / norm
        Ve = ced.view(-1, 1, 1, 1) * R1 * self.hl ** 2
        out["mu_e"] = self.external(self.smooth(prm.cglob * torch.minimum(Ve, beta.view(-1, 1, 1, 1))))
        if prm.flag_les:
            gu = torch.stack([torch.stack(self.grad(c)) for c in ue])  # gu[c][r] = du_c / dx_r
            al = (gu * gu).sum((0, 1))
            V = torch.einsum("caekji,cbekji->abekji", gu, gu) * self.gpv ** (2.0 / 3.0)
            B = V[0, 0] * V[1, 1] + V[0, 0] * V[2, 2] + V[1, 1] * V[2, 2] - V[0, 1] ** 2 - V[0, 2] ** 2 - V[1, 2] ** 2
            m = torch.where(al > 1e-10, prm.c_sgs * torch.sqrt(B.clamp(min=1e-10) / al), self.internal(mus))
            mus = self.external(self.smooth(m))
            out["mu_sgs"] = mus
        L3 = top(torch.stack([c.abs() for c in ue]).amax(0) + self.at(cs))
        mu = self.at(out["mu_fluid"]) / re + (self.internal(mus) if prm.flag_les else 0.0)
        h = self.he / 7.0
        out["dt"] = torch.minimum(prm.cfl_conv * h / L3, prm.cfl_diff * h * h / top(mu)).amin().reshape(1)
        return out

    def steps(self, out, mf, nsteps):
        for _ in range(nsteps):
            y, reta = self.advance([out["rho"], *out["q"], out["E"]], out["dt"], mf, out["mu_e"], out.get("mu_sgs"))
            out = self.closure(y, reta, mf, out.get("mu_sgs"))
        return out

    def laplace(self, x):
        x = x.clone()
        x[0] = 0.0
        y = self.scatter(self.weak_div(self.grad(self.at(x))))
        y[0] = 0.0
        return y

    def laplace_diag(self):
        D2, out = self.D, torch.zeros(self.E, 4, 4, 4, dtype=torch.float64, device="cuda")
        met = [[self.gpv * sum(self.H[c][r] * self.H[c][s] for c in range(3)) for s in range(3)] for r in range(3)]
        out = out + torch.einsum("mi,ekjm->ekji", D2 * D2, met[0][0]) + torch.einsum("mj,ekmi->ekji", D2 * D2, met[1][1]) + \
            torch.einsum("mk,emji->ekji", D2 * D2, met[2][2])
        dg = torch.diagonal(D2)
        di, dj, dk = dg.view(1, 1, 1, 4), dg.view(1, 1, 4, 1), dg.view(1, 4, 1, 1)
        out = out + 2.0 * (met[0][1] * di * dj + met[0][2] * di * dk + met[1][2] * dj * dk)
        return self.scatter(out)


def _exact_rollout(ref, s, case):
    cur = dict(rho=s.rho, q=s.q, E=s.E, mu_e=s.mu_e, dt=s.dt)
    if ref.prm.flag_les:
        cur["mu_sgs"] = s.mu_sgs
    trail = []
    with torch.no_grad():
        for _ in range(case["steps"]):
            trail.append(cur)
            cur = ref.steps(cur, s.mu_factor, 1)
    bar = [torch.zeros_like(s.rho), *cur["q"], torch.zeros_like(s.rho)]
    for c in reversed(trail):
        x = [t.detach().clone().requires_grad_(True) for t in (c["rho"], *c["q"], c["E"])]
        y, _ = ref.advance(x, c["dt"], s.mu_factor, c["mu_e"], c.get("mu_sgs"))
        bar = torch.autograd.grad(y, x, bar)
    return [cur["rho"], cur["q"], cur["E"]], [bar[0], torch.stack(bar[1:4]), bar[4]]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        prm, boxes, states, dts = _members(case, seed)
        outs = []
        for b, h, dt in zip(boxes, states, dts):
            dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
            cur = dict(rho=dev(h.rho), q=dev(h.q), E=dev(h.E), mu_e=dev(h.mu_e), dt=torch.tensor([dt], dtype=torch.float64).cuda())
            outs.append(_Ref(b, prm).steps(cur, dev(h.mu_factor), case["steps"]))
        host = lambda t: t.cpu().numpy().T
        out = {f: np.concatenate([host(o[f]) for o in outs]) for f in STATE}
        out["dt"] = np.array([float(o["dt"]) for o in outs])
        return out
    box, prm, s = _state(case, seed)
    ref = _Ref(box, prm)
    les = prm.flag_les
    if kind in ("step", "steps"):
        cur = dict(rho=s.rho, q=s.q, E=s.E, mu_e=s.mu_e, dt=s.dt)
        if les:
            cur["mu_sgs"] = s.mu_sgs
        out = ref.steps(cur, s.mu_factor, case["steps"])
        return {f: out[f] for f in STATE + (("mu_sgs",) if les else ()) + ("dt",)}
    if kind == "rhs":
        r = ref.rhs(s.rho, s.q, s.E, s.mu_factor, s.mu_e)
        return dict(Rmass=r[0], Rmom=torch.stack(r[1:4]), Rener=r[4], Reta=r[5])
    if kind == "vjp":
        b = _seeds(box, seed)
        x = [t.clone().requires_grad_(True) for t in (s.rho, *s.q, s.E)]
        g = torch.autograd.grad(ref.rhs(x[0], x[1:4], x[4], s.mu_factor, s.mu_e, eta=False), x, list(b))
        return g[0], torch.stack(g[1:4]), g[4]
    if kind == "routines":
        u, q, r = [ref.at(c) for c in s.u], [ref.at(c) for c in s.q], ref.at(s.rho)
        con = [ref.scatter(t) for t in ref.convec(u, q, r, ref.at(s.pr), ref.at(s.e_int))]
        mue = ref.internal(s.mu_e)
        dif = [ref.scatter(t) for t in ref.diffusion(r, u, ref.at(s.Tem), ref.at(s.mu_fluid), mue, torch.zeros_like(mue))]
        pack = lambda t: (t[0], torch.stack(t[1:4]), t[4])
        return pack(con), pack(dif), ref.scatter(ref.scalar(ref.at(s.eta), u, q))
    if kind == "pcg":
        b = _seeds(box, seed)[0]
        b = b - b.mean()
        b[0] = 0.0
        Mi = 1.0 / ref.laplace_diag()
        x, r = torch.zeros_like(b), b.clone()
        z = r * Mi
        p, rz = z.clone(), torch.dot(r, z)
        stop = 1e-13 * b.norm()
        for it in range(40 * case["n"] + 400):
            Ap = ref.laplace(p)
            al = rz / torch.dot(p, Ap)
            x, r = x + al * p, r - al * Ap
            z = r * Mi
            rz, old = torch.dot(r, z), rz
            p = z + rz / old * p
            if it % 32 == 0 and bool(r.norm() < stop):
                break
        return x
    y0 = dict(case)
    s.mu_e.zero_(); s.mu_sgs.zero_()
    return _exact_rollout(ref, s, y0)
