"""The viscous, heat-flux and momentum transport terms of the mixed right-hand side by themselves, against
the FP64 path (1e-12 of the oracle): on the whole residual of a vortex the other terms hide them.

Bound of the viscous and heat terms: a second derivative assembled from FP32 fluxes.  Each flux carries about ten roundings (gradient,
metric, viscosity, gpvol, weak-divergence weights and sums) of 0.3 * 2^-24 rms that add like a random walk;
the weak divergence (row norm 5.3 of D, 2/h = n/pi) raises them against the result, a factor k of the
wave number smaller.  A 5% jitter of the nodes and unequal rows of D: half as much again.  Gradients of
deviations that keep their linear part in FP32 exceed it: those lose the ratio of a field's variation over
the element to its curvature.

Bound of the momentum transport of a shear (whose three directions cancel): one rounding, 0.3 * 2^-24 rms,
of each direction's product at the full scale rho u du/dy."""
import math

import numpy as np
import pytest

from _util import rel_l2, t2n

pytestmark = pytest.mark.gpu


def bound(n, k):
    return 1.5 * math.sqrt(10.0) * 0.3 * 2.0**-24 * (1.0 + 5.3 * n / (math.pi * k))


@pytest.fixture(scope="module")
def mods():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    return torch, M, S


def residuals(mods, n, rho, u, p, mu_factor, mu_e):
    """mixed and FP64 stage residuals of the state (functions of the node coordinates)"""
    torch, M, S = mods
    m = M.periodic_box(n, jitter=0.05, seed=11)
    prm = M.TGVParams()
    gm, s = S.Sod2dMesh(m, prm), S.Sod2dState(m.npoin, m.nelem)
    rho, u, p = (f(*m.coord.T) for f in (rho, u, p))
    for t, a in ((s.rho, rho), (s.u, u.T), (s.q, (rho[:, None] * u).T),
                 (s.E, p / (prm.gamma_gas - 1.0) + 0.5 * rho * (u * u).sum(axis=1))):
        t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    s.mu_factor.fill_(mu_factor)
    s.mu_e.fill_(mu_e)
    out = [gm.rhs(s, precision=q) for q in (S.MIXED, S.FP64)]
    return [{f: t2n(o[f]) for f in ("Rmass", "Rmom", "Rener")} for o in out]


@pytest.mark.parametrize("mu_factor,mu_e", [(1e5, 0.0), (0.0, 1.0)])
@pytest.mark.parametrize("n", [4, 8, 21])
def test_shear(mods, n, mu_factor, mu_e):
    prm = mods[1].TGVParams()
    got, ref = residuals(mods, n, lambda x, y, z: 0 * x + prm.p0 / (prm.Rgas * prm.T0),
                         lambda x, y, z: np.stack([np.sin(y), 0 * y, 0 * y], axis=1), lambda x, y, z: 0 * x + prm.p0,
                         mu_factor * prm.mu_factor, mu_e)
    assert rel_l2(got["Rmom"], ref["Rmom"]) < bound(n, 1.0)


@pytest.mark.parametrize("n", [8, 21])
def test_heat_flux_at_rest(mods, n):
    prm = mods[1].TGVParams()
    got, ref = residuals(mods, n, lambda x, y, z: prm.p0 / (prm.Rgas * (300.0 + 5.0 * np.cos(3.0 * y))),
                         lambda x, y, z: np.zeros((x.size, 3)), lambda x, y, z: 0 * x + prm.p0, 1e4 * prm.mu_factor, 0.0)
    assert rel_l2(got["Rener"], ref["Rener"]) < bound(n, 3.0)


@pytest.mark.parametrize("n", [8, 21, 32])
def test_momentum_transport_of_a_shear(mods, n):
    prm = mods[1].TGVParams()
    rho = prm.p0 / (prm.Rgas * prm.T0)
    got, ref = residuals(mods, n, lambda x, y, z: 0 * x + rho, lambda x, y, z: np.stack([np.sin(y), 0 * y, 0 * y], axis=1),
                         lambda x, y, z: 0 * x + prm.p0, 0.0, 0.0)
    d = got["Rmom"] - ref["Rmom"]
    scale = rho / math.sqrt(8.0)  # rms of rho sin(y) cos(y)
    assert np.linalg.norm(d) / math.sqrt(len(d)) < math.sqrt(3.0) * 0.3 * 2.0**-24 * scale


def test_sgs_viscosity_product(mods):
    """rho mu_sgs enters the stress as one FP64 product rounded once.  Two states with the same velocity,
    pressure, and factors rho and mu_sgs / 4 of 1 and of a value just below the FP32 midpoint 1 + 2^-24.  The
    products are 4 and about 4 (1 + 2^-23), which both round well; FP32 factors would round to 1 and 4 both
    times, and the viscous momentum of the two states would not differ."""
    torch, M, S = mods
    m = M.periodic_box(6, jitter=0.0, seed=0)
    prm = M.TGVParams(flag_les=1)
    gm = S.Sod2dMesh(m, prm)
    u = np.zeros((m.npoin, 3))
    u[:, 0] = np.sin(m.coord[:, 1])
    up = (1.0 + 2.0**-24) * (1.0 - 2.0**-28)
    dt, R = 1e-3, []
    for rho, mus in ((1.0, 4.0), (up, 4.0 * up)):
        s = S.Sod2dState(m.npoin, m.nelem)
        for t, a in ((s.u, u.T), (s.q, (rho * u).T), (s.E, prm.p0 / (prm.gamma_gas - 1.0) + 0.5 * rho * (u * u).sum(axis=1))):
            t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
        s.rho.fill_(rho)
        s.mu_factor.fill_(0.0)
        s.mu_e.fill_(0.0)
        s.mu_sgs.fill_(mus)
        s.dt.fill_(dt)
        stages = torch.empty(15 * m.npoin, dtype=torch.float64, device="cuda")
        q = t2n(s.q)
        gm.rk_4_main_record(s, stages, update_dt=False, precision=S.MIXED)
        R.append((q - t2n(stages[m.npoin:4 * m.npoin].view(3, -1))) * 2.0 / dt)
    # the other roundings are the same in both states or average out over the nodes
    gain = np.vdot(R[1], R[0]) / np.vdot(R[0], R[0]) - 1.0
    assert abs(gain - (up * up - 1.0)) < 2.0**-25, gain
