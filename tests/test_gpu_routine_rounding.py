"""Rounding of the FP64 convection on smooth fields, against the reference's quartets (elem_convec.f90:412-432)
in extended precision on the same metric and inputs.

Bound: with the fields entering the line sums by their differences to the own point, a sum's terms are the
line weights times the nodes' distances (rms 2.5 in xi) of the gradient.  Two roundings of 0.3 * 2^-53 rms each in
three directions: 1.8 * 2^-53 of f |grad u| for one divergence, 1.6 for half the sum of three or a quarter of that of eight; 2
with the metric's.  Whole values in the sums round at |f| / h instead of |grad f|, twice as much on every
refinement."""
import numpy as np
import pytest

from _util import t2n

pytestmark = pytest.mark.gpu
LD = np.longdouble
AXIS = (3, 2, 1)  # fields are [element][k][j][i]


def quartets(D, H, gpv, u, q, rho, pr, E):
    """Element residuals (mass, mom x3, ener) of full_convec_ijk in extended precision."""
    def grad(f):
        g = [np.moveaxis(np.tensordot(D, f, axes=([1], [ax])), 0, ax) for ax in AXIS]
        return [sum(H[c][d] * g[d] for d in range(3)) for c in range(3)]

    def div(f):
        return sum(grad(f[c])[c] for c in range(3))
    k = sum(u[c] * u[c] for c in range(3)) / 2
    dU, dQ, gR, gP = div(u), div(q), grad(rho), grad(pr)
    Rm = (dQ + rho * dU + sum(u[c] * gR[c] for c in range(3))) / 2
    Re = 0
    for f in (E, k):
        gf, grf = grad(f), grad(rho * f)
        Re = Re + (div([rho * f * u[c] for c in range(3)]) + f * dQ + rho * f * dU + rho * div([f * u[c] for c in range(3)])
                   + sum(q[c] * gf[c] + u[c] * grf[c] + f * u[c] * gR[c] for c in range(3))) / 4
    Rmo = []
    for c in range(3):
        gu, gq = grad(u[c]), grad(q[c])
        r = div([q[c] * u[d] for d in range(3)]) + u[c] * dQ + q[c] * dU + rho * div([u[c] * u[d] for d in range(3)])
        Rmo.append((r + sum(u[c] * u[d] * gR[d] + q[d] * gu[d] + u[d] * gq[d] for d in range(3))) / 4 + gP[c])
    return [gpv * r for r in (Rm, *Rmo, Re)]


def geometry(m, gm):
    """Element nodes in i + 4j + 16k order, D, the library's own He and gpvol, and Ml."""
    T, geo = m.tables, gm.geometry()
    order = np.argsort(T.nat_ijk[:, 0] + 4 * T.nat_ijk[:, 1] + 16 * T.nat_ijk[:, 2])
    f = lambda a: a[order].T.reshape(-1, 4, 4, 4).astype(LD)
    H = [[f(geo["He"][c, d]) for d in range(3)] for c in range(3)]
    return m.connec[:, order], np.asarray(T.D).astype(LD), H, f(geo["gpvol"][0]), geo["Ml"]


def assemble(m, conn, r):
    out = np.zeros(m.npoin, dtype=LD)
    np.add.at(out, conn.ravel(), r.ravel())
    return out


@pytest.mark.parametrize("n", [8, 12])
@pytest.mark.parametrize("flow", ["vortex", "shear"])
def test_convection_of_smooth_fields(n, flow):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    m, prm = M.periodic_box(n, jitter=0.05, seed=11), M.TGVParams()
    gm = S.Sod2dMesh(m, prm)
    conn, D, H, gpv, Ml = geometry(m, gm)
    x, y, z = m.coord.T
    if flow == "vortex":
        u = np.stack([np.sin(x) * np.cos(y) * np.cos(z), -np.cos(x) * np.sin(y) * np.cos(z), 0 * x])
        rho = 1.0 + 0.01 * np.cos(2 * x) * np.cos(2 * z)
    else:
        u, rho = np.stack([np.sin(y), 0 * y, 0 * y]), np.ones(m.npoin)
    q, E, pr = rho * u, 180.0 + np.cos(x) * np.cos(y), np.zeros(m.npoin)  # grad p would hide the transport terms
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    Rm, Rmo, Re = gm.full_convec_ijk(dev(u), dev(q), dev(rho), dev(pr), dev(E))
    got = [Rm.cpu().numpy(), *Rmo.cpu().numpy(), Re.cpu().numpy()]
    el = lambda a: a[conn].reshape(-1, 4, 4, 4).astype(LD)
    ref = quartets(D, H, gpv, [el(a) for a in u], [el(a) for a in q], el(rho), el(pr), el(E))
    scale = 1.0 / np.sqrt(2.0)  # rms of |grad u|
    for i, f in ((0, 1.0), (1, 0.5), (2, 0.5), (4, 180.0)):
        err = np.sqrt(np.mean(((got[i] - assemble(m, conn, ref[i])).astype(float) / Ml)**2))
        assert err < 2.0 * 2.0**-53 * f * scale, (i, err / (2.0**-53 * f * scale))


@pytest.mark.parametrize("n", [8, 12])
def test_fused_mass_residual_of_a_shear(n):
    """The FP64 stage residual: div u of the velocity q / rho that the kernel forms itself, on a flow without
    divergence.  The same bound for the mass residual (one divergence)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    m, prm = M.periodic_box(n, jitter=0.05, seed=11), M.TGVParams()
    gm, s = S.Sod2dMesh(m, prm), S.Sod2dState(m.npoin, m.nelem)
    rho = prm.p0 / (prm.Rgas * prm.T0)
    u = np.sin(m.coord[:, 1])
    q = rho * u
    s.rho.fill_(rho)
    s.q.zero_()
    s.q[0].copy_(torch.from_numpy(q))
    s.E.copy_(torch.from_numpy(prm.p0 / (prm.gamma_gas - 1.0) + 0.5 * rho * u * u))
    s.mu_factor.fill_(0.0)
    s.mu_e.fill_(0.0)
    got = t2n(gm.rhs(s, precision=S.FP64)["Rmass"])
    conn, D, H, gpv, Ml = geometry(m, gm)
    el = lambda a: a[conn].reshape(-1, 4, 4, 4).astype(LD)
    Q = [el(q), el(0 * q), el(0 * q)]
    R = LD(rho) + 0 * Q[0]
    ref = assemble(m, conn, quartets(D, H, gpv, [c / R for c in Q], Q, R, 0 * R, 0 * R)[0])
    err = np.sqrt(np.mean((got - (ref / Ml).astype(float))**2))
    assert err < 2.0 * 2.0**-53 * rho / np.sqrt(2.0)


def test_fused_total_enthalpy_energy_of_a_vortex():
    """flag_total_enthalpy differentiates G = E + p.  Bound: u carries one rounding and G two, 0.3 * 2^-53 rms
    each, which the rows of D (norm 3.9 rms) and the element size (n / pi) raise: 3.9 * 0.3 * sqrt(3) of u G n / pi.
    Formed as rho (h + k), G adds the roundings of h, of k, of their sum and of the product."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    n = 8
    m, prm = M.periodic_box(n, jitter=0.05, seed=11), M.TGVParams(flag_total_enthalpy=1)
    gm, s = S.Sod2dMesh(m, prm), S.Sod2dState.from_host(M.taylor_green_state(m, prm, 1e-2, seed=4), m.nelem)
    s.mu_factor.fill_(0.0)
    s.mu_e.fill_(0.0)
    got = t2n(gm.rhs(s, precision=S.FP64)["Rener"])
    conn, D, H, gpv, Ml = geometry(m, gm)
    el = lambda t: t.cpu().numpy()[conn].reshape(-1, 4, 4, 4).astype(LD)
    rho, q, E, g = el(s.rho), [el(s.q[c]) for c in range(3)], el(s.E), LD(prm.gamma_gas)
    u = [c / rho for c in q]
    G = E + (g - 1) * (E - rho * sum(c * c for c in u) / 2)

    def grad(f):
        d = [np.moveaxis(np.tensordot(D, f, axes=([1], [ax])), 0, ax) for ax in AXIS]
        return [sum(H[c][k] * d[k] for k in range(3)) for c in range(3)]
    div = lambda f: sum(grad(f[c])[c] for c in range(3))
    ref = assemble(m, conn, gpv * (div([G * c for c in u]) + G * div(u) + sum(c * d for c, d in zip(u, grad(G)))) / 2) / Ml
    err = np.sqrt(np.mean((got - ref).astype(float)**2))
    uG = float(np.sqrt(np.mean(sum(c * c for c in u))) * np.mean(G))
    assert err < 3.9 * 0.3 * np.sqrt(3.0) * 2.0**-53 * uG * n / np.pi
