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
