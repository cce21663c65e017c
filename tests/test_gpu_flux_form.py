"""The fused element RHS kernels on states that vary strongly inside an element (density by a
factor of 3, pressure by 6, velocity of the size of the sound speed), where every second-order
term of their two-point flux sums is of leading order: each elements-per-CTA configuration (27
elements: partial tiles at 2, 4 and 8), both energy forms, with and without the SGS viscosity,
against the oracle's stage residual.

Bounds: FP64 1e-12 (the FP64 path's bound).  Mixed: a residual is a sum of products of up to four
FP32 factors (metric, line weight, mean velocity, mean density) with a difference, about 6
roundings of 2^-24 per term and 12 terms per sum that add like a random walk at most doubled by
the cancellation of these states: 2^-24 * 6 * sqrt(12) = 1.2e-6 per field.
"""
import dataclasses

import numpy as np
import pytest

from _util import rel_l2, t2n

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(oracle):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    m = M.periodic_box(3, jitter=0.05, seed=9)
    prm = M.TGVParams()
    st = M.taylor_green_state(m, prm, pert_amp=1e-2, seed=9)
    x, y, z = (m.coord[:, c] for c in range(3))
    rho = 1.0 + 0.5 * np.sin(x) * np.cos(2 * y + z)
    p = 10.0 * np.exp(0.9 * np.sin(2 * x - z) * np.cos(y))
    u = np.stack([3.0 * np.sin(x + y), 2.0 * np.cos(z - x), 4.0 * np.sin(2 * y) * np.cos(z)], axis=1)
    g = prm.gamma_gas
    st.rho = rho
    st.u = np.asfortranarray(u)
    st.q = np.asfortranarray(rho[:, None] * u)
    st.E = p / (g - 1.0) + 0.5 * rho * (u * u).sum(axis=1)
    st.mu_factor = np.full(m.npoin, 1e3 * prm.mu_factor)
    rng = np.random.default_rng(9)
    st.mu_e = np.asfortranarray(0.05 * rng.random((m.nelem, 64)))
    return dict(M=M, S=S, m=m, prm=prm, om=oracle.OracleMesh(m), st=st)


@pytest.mark.parametrize("toth", [0, 1])
@pytest.mark.parametrize("epb", [1, 2, 4, 8])
def test_stage_residual(env, oracle, toth, epb):
    S, st = env["S"], env["st"]
    prm = dataclasses.replace(env["prm"], flag_total_enthalpy=toth)
    ref = oracle.rk4(env["om"], prm, st.copy(), 1e-6, nsteps=1, capture_stage=1)
    gm = S.Sod2dMesh(env["m"], prm)
    s = S.Sod2dState.from_host(st, gm.nelem)
    for prec, tol in ((S.FP64, 1e-12), (S.MIXED, 1.2e-6)):
        gm.set_rhs_config(prec, epb)
        out = gm.rhs(s, precision=prec)
        for k in ("Rmass", "Rmom", "Rener", "Reta"):
            err = rel_l2(t2n(out[k]), ref[k])
            assert err < tol, (prec, k, err)
