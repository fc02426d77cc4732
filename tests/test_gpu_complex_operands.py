"""Mixed solves whose tensor-core operands are complex: one gather fills the tiles of both
components from the packed split."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,A,snm,theta", [
    (1, 4, True, (0.0, 0.0, 0.0)),    # blocks far below one tile
    (1, 14, False, (0.4, -0.9, 1.7)),  # a twist: channels of every size, odd ones included
    (1, 28, True, (0.0, 0.0, 0.0)),
    (2, 28, True, (0.3, 1.1, -0.6)),   # several row and K tiles an operand
])
@pytest.mark.parametrize("prec,rebase", [("PREC_MIXED", "REBASE_DIGITS"), ("PREC_MIXED_TF32", "REBASE_FP64")])
def test_complex_operands(ccx, nmax, A, snm, theta, prec, rebase):
    """The converged energy of the FP64 solve: both stop at a residual norm below 1e-10, and
    the the energy moves by the potential (tens of MeV) times the difference of the amplitudes: 1e-9."""
    L = ccx.Layout.from_basis(nmax, A, 0.16 if snm else 0.08, snm=snm, theta=theta)
    res = []
    for p, kw in ((ccx.PREC_FP64, {}), (getattr(ccx, prec), dict(rebase=getattr(ccx, rebase)))):
        e = ccx.Engine(L, real=False)
        e.generate(potential=ccx.POT_CHIRAL_LIKE)
        e.setup_t_amplitudes()
        res.append(e.ccd_iter(mode=ccx.MODE_STANDARD, precision=p, tol=1e-10, max_iter=200, **kw))
        e.close()
    r64, rm = res
    assert r64["converged"] and rm["converged"]
    assert abs(rm["e_ccd"] - r64["e_ccd"]) < 1e-9 * abs(r64["e_ccd"])
