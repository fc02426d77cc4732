"""(T) of lattices that give a thread block less than two items of the usual split (every nseg-th
test instead), and hole triples on one momentum, taken as single pairs by FP64 contractions.

Tolerances as for the momentum blocks: 1e-10 of E(T) for FP64 contractions in another order than
the oracle's, 1e-5 for FP32."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmax,A,pot,real,theta", [
    (2, 4, 1, False, (0.0, 0.0, 0.0)),    # one hole momentum, many particle momenta
    (2, 3, 1, False, (0.2, -0.1, 0.4)),   # partly filled: one hole triple
    (1, 28, 0, True, (0.0, 0.0, 0.0)),    # real, several hole momenta
    (1, 12, 0, True, (0.3, 0.5, -0.2)),
    (1, 16, 1, False, (0.0, 0.0, 0.0)),
])
def test_triples_of_small_lattices(ccx, O, nmax, A, pot, real, theta):
    o = O.Oracle(O.Config(nmax=nmax, A=A, rho=0.16, snm=True, theta=theta, potential=pot))
    e = ccx.Engine(ccx.Layout.from_basis(nmax, A, 0.16, snm=True, theta=theta), real=real)
    e.generate(potential=pot)
    o.mp2()
    e.setup_t_amplitudes()
    want = o.triples()
    got32 = e.pert_triples()
    e.set_triples_precision(fp32=False)
    got = e.pert_triples()
    assert abs(got - want) <= 1e-10 * abs(want), (got, want)
    assert abs(got32 - want) <= 1e-5 * abs(want), (got32, want)
    o.close()
    e.close()
