"""Rounding of full_convec_ijk on smooth fields, against the reference's quartets (elem_convec.f90:412-432)
in extended precision on the same metric and inputs.

Bound: with the fields entering the line sums by their differences to the own point, a sum's terms are the
line weights times the nodes' distances (rms 2.5 in xi) of the gradient.  Two roundings of 0.3 * 2^-53 rms each in
three directions: 1.8 * 2^-53 of f |grad u| for one divergence, 1.6 for half the sum of three or a quarter of that of eight; 2
with the metric's.  Whole values in the sums round at |f| / h instead of |grad f|, twice as much on every
refinement."""
import numpy as np
import pytest

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


@pytest.mark.parametrize("n", [8, 12])
@pytest.mark.parametrize("flow", ["vortex", "shear"])
def test_convection_of_smooth_fields(n, flow):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    m, prm = M.periodic_box(n, jitter=0.05, seed=11), M.TGVParams()
    gm, T = S.Sod2dMesh(m, prm), m.tables
    order = np.argsort(T.nat_ijk[:, 0] + 4 * T.nat_ijk[:, 1] + 16 * T.nat_ijk[:, 2])
    conn, geo = m.connec[:, order], gm.geometry()
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
    H = [[geo["He"][c, d][order].T.reshape(-1, 4, 4, 4).astype(LD) for d in range(3)] for c in range(3)]
    gpv = geo["gpvol"][0][order].T.reshape(-1, 4, 4, 4).astype(LD)
    ref = quartets(np.asarray(T.D).astype(LD), H, gpv, [el(a) for a in u], [el(a) for a in q], el(rho), el(pr), el(E))
    scale = 1.0 / np.sqrt(2.0)  # rms of |grad u|
    for i, f in ((0, 1.0), (1, 0.5), (2, 0.5), (4, 180.0)):
        r = np.zeros(m.npoin, dtype=LD)
        np.add.at(r, conn.ravel(), ref[i].ravel())
        err = np.sqrt(np.mean(((got[i] - r).astype(float) / geo["Ml"])**2))
        assert err < 2.0 * 2.0**-53 * f * scale, (i, err / (2.0**-53 * f * scale))
