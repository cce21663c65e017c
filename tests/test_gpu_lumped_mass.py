"""The lumped mass a caller hands over with the mesh."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sod2d_refmap_b200 import build, mesh as M, solver as S
    build.build()
    return torch, M, S


@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
def test_zero_on_a_working_row_is_not_hidden(mods, precision):
    """A zero lumped mass divides, as in lumped_solver: the row's residual is not finite and the step raises
    the flag, instead of leaving the node frozen."""
    torch, M, S = mods
    prec = getattr(S, precision)
    m, prm = M.periodic_box(3, jitter=0.05, seed=1), M.TGVParams()
    ml = S.Sod2dMesh(m, prm).geometry()["Ml"]
    ml[7] = 0.0
    gm = S.Sod2dMesh(m, prm, geometry={"Ml": ml})
    s = S.Sod2dState.from_host(M.taylor_green_state(m, prm), gm.nelem)
    s.dt.fill_(1e-3)
    out = gm.rhs(s, precision=prec)
    for f in ("Rmass", "Rener"):
        bad = ~torch.isfinite(out[f])
        assert bool(bad[7]) and int(bad.sum()) == 1, f
    R = torch.ones(m.npoin, dtype=torch.float64, device="cuda")
    gm.lumped_solver(R)
    assert not bool(torch.isfinite(R[7]))
    gm.rk_4_main(s, precision=prec)
    with pytest.raises(RuntimeError):
        gm.check_finite()
    assert not bool(torch.isfinite(s.rho[7]))


def test_first_call_launches_no_more_than_the_second(mods):
    """What depends on the mesh alone is formed with the handle: the FP64 right-hand side, its adjoint and a routine."""
    torch, M, S = mods
    from sod2d_refmap_b200 import _lib
    m, prm = M.periodic_box(3, jitter=0.05, seed=1), M.TGVParams()
    st = M.taylor_green_state(m, prm)
    calls = (lambda g, s: g.rhs(s, precision=S.FP64),
             lambda g, s: g.rhs_vjp(s.rho, s.q, s.E, s.mu_e, s.mu_factor, s.rho, s.q, s.E),
             lambda g, s: g.full_convec_ijk(s.u, s.q, s.rho, s.pr, s.E))
    for call in calls:
        gm = S.Sod2dMesh(m, prm)
        s = S.Sod2dState.from_host(st, gm.nelem)
        counts = [_lib.launch_count()]
        for _ in range(2):
            call(gm, s)
            counts.append(_lib.launch_count())
        assert counts[1] - counts[0] == counts[2] - counts[1]
