"""Branches of the kernels' launch rules at the sizes where they change: the Poisson node kernels in
one trip and grid-stride, ensemble members beyond one chunk round of the entropy statistics, the
stage-4 entropy sums within and beyond one wave of blocks, the shock sensor on both sides of its cap, and
the per-routine kernels on unrelated u, q and E.

Bounds: 1e-12 relative per field, the FP64 path's bound (each compares sums of the same terms in
another order)."""
import numpy as np
import pytest

from _util import rel_l2, t2n

pytestmark = pytest.mark.gpu

TOL64 = 1e-12


@pytest.fixture(scope="module")
def mods():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    return torch, M, S


def dev(torch, a):
    a = np.asarray(a)
    return torch.from_numpy(np.ascontiguousarray(a.T if a.ndim == 2 else a)).cuda()


def laplace_numpy(m, x):
    """eval_laplacian_mult by dense einsums: sum_dir D^T (gpvol He^T He D x), node 0 pinned."""
    T = m.tables
    order = np.argsort(T.nat_ijk[:, 0] + 4 * T.nat_ijk[:, 1] + 16 * T.nat_ijk[:, 2])
    conn, orig = m.connec[:, order], m.connec_orig[:, order]
    from sod2d_refmap_b200.mesh import gll_nodes_weights
    D, w = T.D, gll_nodes_weights()[1]
    iso = lambda f: np.stack([np.einsum("im,ekjm->ekji", D, f), np.einsum("jm,ekmi->ekji", D, f),
                              np.einsum("km,emji->ekji", D, f)])
    J = np.stack([iso(m.coord_orig[:, c][orig].reshape(-1, 4, 4, 4)) for c in range(3)])  # [c][r]
    Jm = np.moveaxis(J, (0, 1), (-2, -1))
    He = np.moveaxis(np.linalg.inv(Jm), (-2, -1), (0, 1))  # [r][c] = dxi_r / dx_c
    gpv = w[:, None, None] * w[None, :, None] * w[None, None, :] * np.linalg.det(Jm)
    x = x.copy()
    x[0] = 0.0
    g = iso(x[conn].reshape(-1, 4, 4, 4))
    grad = [sum(He[r][c] * g[r] for r in range(3)) for c in range(3)]
    F = [gpv * sum(He[r][c] * grad[c] for c in range(3)) for r in range(3)]
    R = (np.einsum("mi,ekjm->ekji", D, F[0]) + np.einsum("mj,ekmi->ekji", D, F[1]) +
         np.einsum("mk,emji->ekji", D, F[2]))
    y = np.bincount(conn.ravel(), weights=R.ravel(), minlength=m.npoin)
    y[0] = 0.0
    return y


@pytest.mark.parametrize("n", [3, 10, 29])  # 729, 27,000 and 658,503 nodes (the last grid-stride)
def test_poisson_product_and_solve(mods, n):
    torch, M, S = mods
    m = M.periodic_box(n, jitter=0.05, seed=n)
    P = S.Sod2dPoisson(S.Sod2dMesh(m, M.TGVParams()))
    rng = np.random.default_rng(n)
    x = rng.standard_normal(m.npoin)
    assert rel_l2(P.apply(torch.from_numpy(x).cuda()).cpu().numpy(), laplace_numpy(m, x)) < TOL64
    b = rng.standard_normal(m.npoin)
    b -= b.mean()
    for mixed in (False, True):
        sol, it, rel = P.solve(torch.from_numpy(b).cuda(), tol=1e-9, mixed=mixed)
        b0 = b.copy()
        b0[0] = 0.0
        # the true residual: the solver's own recursion stopped below 1e-9
        assert rel < 1e-9
        assert np.linalg.norm(laplace_numpy(m, sol.cpu().numpy()) - b0) < 2e-9 * np.linalg.norm(b0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ensemble_members_beyond_one_chunk_round(mods, precision):
    """Members of 9,261 and 729 nodes (32 chunks of 256 nodes hold 8,192) against the meshes alone."""
    torch, M, S = mods
    prec = S.FP64 if precision == "fp64" else S.MIXED
    prm = M.TGVParams()
    boxes = [M.periodic_box(7, jitter=0.05, seed=2), M.periodic_box(3, jitter=0.05, seed=3)]
    states = [M.taylor_green_state(b, prm, 1e-2, seed=i) for i, b in enumerate(boxes)]
    batch = S.Sod2dBatch(boxes, states, prm)
    dts = [2e-3, 4e-3]
    batch.set_dt(dts)
    batch.rk4_steps(3, prec)
    for i, (b, st, dt) in enumerate(zip(boxes, states, dts)):
        gm = S.Sod2dMesh(b, prm)
        s = S.Sod2dState.from_host(st, gm.nelem)
        s.dt.fill_(dt)
        gm.rk4_steps(s, 3, prec)
        got, ref = batch.get_member(i), s.to_host()
        # mixed: mu_e differs in the last bits (blocking of the entropy sums) and is then rounded to
        # FP32 for the next step, 2^-24 of a term that is a hundredth of the residual at most
        tol = TOL64 if prec == S.FP64 else 1e-9
        for f in ("rho", "q", "E", "mu_e", "Reta"):
            assert rel_l2(got[f], ref[f]) < tol, (i, f)
        assert abs(batch.dt()[i] - float(s.dt.item())) <= tol * dt


@pytest.mark.parametrize("speed", [0.3, 8.0, 14.0])  # element Mach numbers up to ~0.03, 0.8 and 1.4
def test_shock_sensor_both_sides_of_its_cap(mods, oracle, speed):
    torch, M, S = mods
    m = M.periodic_box(3, jitter=0.05, seed=4)
    prm = M.TGVParams()
    st = M.taylor_green_state(m, prm, 1e-2, seed=4)
    st.u *= speed
    rng = np.random.default_rng(4)
    Reta = rng.standard_normal(m.npoin)
    ref = oracle.smart_visc(oracle.OracleMesh(m), prm, Reta, st.rho, st.u, st.csound, st.Tem, st.eta,
                            np.zeros((m.nelem, 64), order="F"))
    gm = S.Sod2dMesh(m, prm)
    got = gm.smart_visc_spectral(*(dev(torch, a) for a in (Reta, st.rho, st.u, st.csound, st.Tem, st.eta)))
    assert rel_l2(t2n(got), ref) < TOL64


@pytest.mark.parametrize("n", [1, 3])
def test_routines_on_unrelated_fields(mods, oracle, n):
    """q is not rho u and E is not the state's: every product of the quartets is on its own."""
    torch, M, S = mods
    m = M.periodic_box(n, jitter=0.05 if n > 1 else 0.0, seed=5)
    prm = M.TGVParams()
    om, gm = oracle.OracleMesh(m), S.Sod2dMesh(m, prm)
    rng = np.random.default_rng(5)
    N = m.npoin
    u, q = (np.asfortranarray(rng.standard_normal((N, 3))) for _ in range(2))
    rho, pr, E, eta, Tem, muf = (1.0 + rng.random(N) for _ in range(6))
    mue, mus = (np.asfortranarray(rng.random((m.nelem, 64))) for _ in range(2))
    d = lambda a: dev(torch, a)
    for got, ref in ((gm.full_convec_ijk(d(u), d(q), d(rho), d(pr), d(E)), oracle.convec(om, u, q, rho, pr, E)),
                     (gm.full_convec_ijk_H(d(u), d(q), d(rho), d(pr), d(E)), oracle.convec_H(om, u, q, rho, pr, E)),
                     (gm.full_diffusion_ijk(d(rho), d(E), d(u), d(Tem), d(muf), d(mue), d(mus)),
                      oracle.diffusion(om, prm, rho, E, u, Tem, muf, mue, mus))):
        for g, r in zip(got, ref):
            assert rel_l2(t2n(g), r) < TOL64
    assert rel_l2(t2n(gm.generic_scalar_convec_ijk(d(q), d(eta), d(u))), oracle.scalar_convec(om, q, eta, u)) < TOL64


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [17, 18])  # 519 and 616 blocks of the stage-4 gather: within and beyond one wave of 4 x 148
def test_entropy_normalisation_around_one_wave(mods, n, precision):
    """The step's mean and norm of the entropy (formed by the gather's last block, or by a launch of their
    own) against smart_visc_spectral on the fields the step left, whose norm comes from another kernel."""
    torch, M, S = mods
    m, prm = M.periodic_box(n, jitter=0.05, seed=6), M.TGVParams()
    gm = S.Sod2dMesh(m, prm)
    s = S.Sod2dState.from_host(M.taylor_green_state(m, prm, 1e-2, seed=6), gm.nelem)
    s.dt.fill_(1e-3)
    gm.rk_4_main(s, S.FP64 if precision == "fp64" else S.MIXED)
    ref = gm.smart_visc_spectral(s.Reta, s.rho, s.u, s.csound, s.Tem, s.eta)
    spread = float((s.eta - s.eta.mean()).abs().max() / s.eta.abs().max())
    # the norm is a difference of FP64 sums of N terms: N^(1/2) roundings of the mean against the spread
    assert rel_l2(t2n(s.mu_e), t2n(ref)) < 4 * m.npoin**0.5 * 2.0**-53 / spread
